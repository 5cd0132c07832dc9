"""The exact Guevel-Delhommeau term's closed form (csrc/mh_egd.cuh) against the oracle's
adaptive quadrature of exact_Guevel_Delhommeau.jl:15-46, at the edges of its rules: the power
series (r < 3 and r < Y/2, up to min(Y, 3)), the two Gauss-Legendre rules (lengths 22 and 38),
the Bessel tables' end (r = 8), r = 0, and the points it leaves to the quadrature (z > 0)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

RTOL, ATOL = 1e-12, 1e-14  # the oracle's quadrature of the quarter integral (the term is four times it)


def _check(mh, oracle, ctx, r, z):
    got = mh._device.exact_wave_terms(ctx, r, z, rtol=RTOL, atol=ATOL)
    for i, (a, b) in enumerate(zip(r, z)):
        ref = oracle.egd_dimless(a, b, RTOL, ATOL), oracle.egd_dimless_dr(a, b, RTOL, ATOL)
        for g, want in zip(got[i], ref):
            # the oracle's own tolerance, and 50 roundings of the term's scale |G| + 2/d
            bound = RTOL * abs(want) + 4 * ATOL + 50 * 2.0 ** -53 * (abs(want) + 2 / np.hypot(a, b))
            assert abs(g - want) <= bound, (a, b, g, want, abs(g - want), bound)


@pytest.mark.parametrize("Y", [1e-3, 0.7, 2.9999, 3.0001, 5.99, 6.01, 21.9, 22.1, 24.9, 25.1, 37.9, 38.1, 41.2, 70.0])
def test_closed_form_at_rule_edges(mh, oracle, ctx, Y):
    r = [0.0, 1e-9 * Y, 1e-3 * Y, 0.4999 * Y, 0.5001 * Y, Y, 2.9999, 3.0001, 7.9999, 8.0001, 30.0]
    _check(mh, oracle, ctx, np.array(r), np.full(len(r), -Y))


def test_closed_form_over_the_range(mh, oracle, ctx):
    rng = np.random.default_rng(12)
    _check(mh, oracle, ctx, 10 ** rng.uniform(-6, 2, 200), -10 ** rng.uniform(-4, 1.8, 200))


def test_points_above_the_surface_take_the_quadrature(mh, oracle, ctx):
    r = np.array([0.0, 0.3, 2.0, 9.0])
    _check(mh, oracle, ctx, r, np.array([0.5, 0.1, 1.5, 0.02]))


@pytest.mark.parametrize("n_lat", [3, 7, 13])  # 18, 98 and 338 panels: ragged row and column tiles
@pytest.mark.parametrize("direct", [True, False])
def test_exact_assembly_of_ragged_sizes(mh, oracle, ctx, n_lat, direct):
    mesh = mh.hemisphere_mesh(1.7, n_lat, 2 * n_lat)
    S, D = mh.assemble_matrices(mh.default_greens_functions("ExactGuevelDelhommeau"), mesh, 0.9, direct=direct, ctx=ctx)
    oracle.set_egd_tolerance(RTOL, ATOL)
    So, Do = oracle.assemble_matrices(mesh, 0.9, gfs=oracle.DEFAULT_EGD, direct=direct)
    # entries carry the quadrature's 1e-12 relative and 4e-14 absolute of terms of order one
    assert np.linalg.norm(S - So) <= 2e-12 * np.linalg.norm(So)
    assert np.linalg.norm(D - Do) <= 2e-12 * np.linalg.norm(Do)
