"""The exact Guevel-Delhommeau term's closed form (csrc/mh_egd.cuh) against the oracle's
adaptive quadrature of exact_Guevel_Delhommeau.jl:15-46, at the edges of its rules: the power
series (r < 3 and r < Y/2, up to min(Y, 3)), the two Gauss-Legendre rules (lengths 22 and 38),
the Bessel tables' end (r = 8), r = 0, and the points it leaves to the quadrature (z > 0)."""
import time

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


def test_points_above_the_surface_go_to_whole_warps(mh, ctx):
    # 256 points one warp each take 1.7 ms; one thread each, 280 ms
    rng = np.random.default_rng(3)
    r, z = rng.uniform(0.1, 60, 256), rng.uniform(0.01, 2, 256)
    mh._device.exact_wave_terms(ctx, r, z)
    times = []
    for _ in range(3):
        t0 = time.perf_counter()
        mh._device.exact_wave_terms(ctx, r, z)
        times.append(time.perf_counter() - t0)
    assert min(times) < 0.05, times


def test_mixed_and_non_finite_points(mh, oracle, ctx):
    # points of both kinds side by side (ragged warps and CTAs), and not a number where one goes in
    rng = np.random.default_rng(4)
    r, z = rng.uniform(0.1, 9, 301), rng.uniform(-2, 0.5, 301)
    _check(mh, oracle, ctx, r, z)
    r[[3, 140]], z[[7, 299]] = [np.nan, np.inf], [np.nan, -np.inf]
    got = mh._device.exact_wave_terms(ctx, r, z)
    bad = np.zeros(301, bool)
    bad[[3, 7, 140, 299]] = True
    assert np.isnan(got[bad]).all() and np.isfinite(got[~bad]).all()


def _raised(mh, mesh, up):
    V = mesh.vertices.copy()
    V[:, 2] += up
    return mh.StaticArraysMesh(V, mesh.faces)


@pytest.mark.parametrize("n_lat", [3, 7])
@pytest.mark.parametrize("up", [0.4, 1.9])  # partly and wholly above the surface
@pytest.mark.parametrize("direct", [True, False])
def test_exact_assembly_above_the_surface(mh, oracle, ctx, n_lat, up, direct):
    mesh = _raised(mh, mh.hemisphere_mesh(1.7, n_lat, 2 * n_lat), up)
    S, D = mh.assemble_matrices(mh.default_greens_functions("ExactGuevelDelhommeau"), mesh, 0.9, direct=direct, ctx=ctx)
    oracle.set_egd_tolerance(RTOL, ATOL)
    So, Do = oracle.assemble_matrices(mesh, 0.9, gfs=oracle.DEFAULT_EGD, direct=direct)
    assert np.linalg.norm(S - So) <= 2e-12 * np.linalg.norm(So)
    assert np.linalg.norm(D - Do) <= 2e-12 * np.linalg.norm(Do)


def test_both_wave_terms_above_the_surface(mh, ctx):
    # Wu and exact term together are the sum of the two (the static part counted once)
    mesh = _raised(mh, mh.hemisphere_mesh(1.7, 5, 10), 0.4)
    rankine = (mh.Rankine(), mh.RankineReflected())
    sets = (rankine + (mh.GFWu(), mh.ExactGuevelDelhommeau()), rankine + (mh.GFWu(),),
            rankine + (mh.ExactGuevelDelhommeau(),), rankine)
    for direct in (True, False):
        both, wu, exact, static = (np.stack(mh.assemble_matrices(g, mesh, 0.9, direct=direct, ctx=ctx)) for g in sets)
        ok = np.isfinite(wu)  # the fits have no value on the vertical above the surface
        assert ok.mean() > 0.9 and np.array_equal(ok, np.isfinite(both)) and np.isfinite(exact).all()
        # a few roundings of the terms
        scale = np.abs(exact).max() + np.abs(wu[ok]).max() + np.abs(static).max()
        assert np.abs(both - (wu + exact - static))[ok].max() <= 16 * 2.0 ** -53 * scale


def test_frequency_derivative_above_the_surface(mh, ctx):
    # the derivative's pair values: its formula in numpy, from the point evaluator and the matrices
    mesh = _raised(mh, mh.hemisphere_mesh(1.7, 6, 12), 0.3)
    gfs, om, rho, g = mh.default_greens_functions("ExactGuevelDelhommeau"), 1.1, 1000.0, 9.81
    body = mh.FloatingBody(mesh, ["Heave"], body_name="raised")
    out = mh.hydrodynamic_coefficients_derivative(body, {"wave_frequencies": [om], "radiating_dofs": ["Heave"],
                                                         "influenced_dofs": ["Heave"]}, mh.DirectBEM(gfs), ctx=ctx,
                                                  rho=rho, g=g)
    n, k = mesh.nfaces, om ** 2 / g
    S, D = mh.assemble_matrices(gfs, mesh, k, ctx=ctx)
    dx = mesh.centers[None] - mesh.centers[:, None]  # source minus field point
    dis, Z = np.hypot(dx[..., 0], dx[..., 1]), mesh.centers[:, None, 2] + mesh.centers[None, :, 2]
    r, z = k * dis, k * Z
    assert (z > 0).any() and (z < 0).any()
    v = mh._device.exact_wave_terms(ctx, np.ascontiguousarray(r.ravel()), np.ascontiguousarray(z.ravel()))
    G, Gr = v[:, 0].reshape(n, n), np.where(r > 1e-6, v[:, 1].reshape(n, n), 0.0)
    d = np.hypot(r, z)
    Gz = G + 2 / d
    Gzz, Grz = Gz - 2 * z / d ** 3, Gr - 2 * r / d ** 3
    far = r > 1e-6
    Grr = np.where(far, -Gr / np.where(far, r, 1.0) - Gzz, 0.0)
    nj = mesh.normals[None]
    u = np.where(far, (nj[..., 0] * dx[..., 0] + nj[..., 1] * dx[..., 1]) / np.where(far, dis, 1.0), 0.0)
    a, n3 = -mesh.areas[None] / (4 * np.pi), nj[..., 2]
    dS = a * (G + r * Gr + z * Gz)
    dD = a * k * (2 * (u * Gr + n3 * Gz) + u * (r * Grr + z * Grz) + n3 * (r * Grz + z * Gzz))
    nz = mesh.normals[:, 2]
    b, db = -1j * om * nz, -1j * nz
    phi = np.linalg.solve(D, S @ b)
    dphi = np.linalg.solve(D, 2 * om / g * (dS @ b - dD @ phi) + S @ db)
    w = -1j * rho * nz * mesh.areas
    F, dF = om * (w @ phi), w @ phi + om * (w @ dphi)
    # n roundings of a sum and the quadrature's 1e-12 per entry, magnified by the solve
    for got, want in ((out["added_mass"], F.real / om ** 2), (out["radiation_damping"], F.imag / om),
                      (out["d_added_mass"], dF.real / om ** 2 - 2 * F.real / om ** 3),
                      (out["d_radiation_damping"], dF.imag / om - F.imag / om ** 2)):
        assert abs(float(np.ravel(got)[0]) - want) <= 1e-9 * max(abs(F) / om, abs(dF)), (got, want)
