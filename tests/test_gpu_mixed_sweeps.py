"""The FP32 factors, substitutions and residual products of the mixed precision seen by themselves.
When the refinement does not converge, the FP64 factorization gives the answer all the same, so the
solution alone cannot show that one of them is wrong: these tests count the refinement's sweeps and
see that no FP64 panel was factored."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def pctx(mh):
    c = mh.Context(0)
    c.profile(True)
    return c


def _kernels(ctx, call):
    ctx.profile_reset()
    out = call()
    return out, {name: count for name, (_, count) in ctx.profile_read().items()}


def _well_conditioned(n):
    # diagonal 3, the rest a random matrix of spectral radius 1.4: condition below 4
    rng = np.random.default_rng(n)
    A = (rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n))) / np.sqrt(n)
    A[np.arange(n), np.arange(n)] += 3.0
    return A


# a sweep gains at least a factor of 1e5 on these matrices (FP32 rounding 6e-8, condition 4, growth
# of the factors): from 1e-5 to the stopping rule of about 1e-15 in two sweeps, three residuals; one
# more is allowed
SWEEPS = 4


@pytest.mark.parametrize("n", [1, 31, 33, 64, 97, 200, 431, 545, 861, 1041, 1537, 2050, 2900, 3001])
@pytest.mark.parametrize("adjoint", [False, True])
def test_few_sweeps_and_no_fp64_factors(mh, pctx, n, adjoint):
    # 2900 and 3001: the first updates take two panels at once
    A = _well_conditioned(n)
    rng = np.random.default_rng(n + 1)
    b = rng.standard_normal((n, 3)) + 1j * rng.standard_normal((n, 3))
    solve = mh.linsolve_adjoint if adjoint else mh.linsolve
    x, k = _kernels(pctx, lambda: solve(A, b, precision="mixed", ctx=pctx))
    assert k["lu_panel_f32"] > 0 and "lu_panel_f64" not in k and k["ir_norms"] <= SWEEPS, k
    r = np.abs(b - (A.conj().T if adjoint else A) @ x).max(axis=0)
    assert (r <= 20 * n * 2.0 ** -53 * np.abs(A).sum(axis=1).max() * np.abs(x).max(axis=0)).all()


@pytest.mark.parametrize("n, rhs", [(33, 1), (64, 9), (200, 2), (300, 17), (545, 8), (1000, 33), (1537, 5), (2999, 3)])
@pytest.mark.parametrize("adjoint", [False, True])
def test_substitution_shapes_in_fp32(mh, pctx, n, rhs, adjoint):
    A = _well_conditioned(n)
    b = np.random.default_rng(rhs).standard_normal((n, rhs)) + 0j
    solve = mh.linsolve_adjoint if adjoint else mh.linsolve
    _, k = _kernels(pctx, lambda: solve(A, b, precision="mixed", ctx=pctx))
    assert "lu_panel_f64" not in k and k["ir_norms"] <= SWEEPS, k


@pytest.mark.parametrize("n", [97, 545, 1100, 2950])
def test_pivots_from_other_ctas_in_fp32(mh, pctx, n):
    # a permuted well-conditioned matrix: every interchange of the first half takes a row held
    # elsewhere
    A = np.roll(_well_conditioned(n), n // 2, axis=0)
    b = np.random.default_rng(n).standard_normal((n, 2)) + 0j
    _, k = _kernels(pctx, lambda: mh.linsolve(A, b, precision="mixed", ctx=pctx))
    assert "lu_panel_f64" not in k and k["ir_norms"] <= SWEEPS, k


@pytest.mark.parametrize("direct", [True, False])
def test_batch_of_several_orders(mh, pctx, direct):
    # a class of 1230 to 1300 panels with 8 frequencies (two panels per update, matrices that end
    # inside the second) and one of 98; each body ends its refinement by itself
    bodies = [mh.FloatingBody(mh.hemisphere_mesh(1.0, r, c), ["Heave", "Surge"], body_name=f"h{r}")
              for r, c in ((30, 41), (13, 97), (26, 50), (7, 14))]
    p = {"wave_frequencies": np.linspace(0.5, 2.4, 8), "radiating_dofs": ["Heave", "Surge"],
         "influenced_dofs": ["Heave", "Surge"], "wave_directions": [0.3]}
    F = (mh.DirectBEM if direct else mh.IndirectBEM)(precision="mixed")
    _, k = _kernels(pctx, lambda: mh.batch_hydrodynamic_coefficients(bodies, [p] * 4, F, ctx=pctx, rho=1025.0))
    assert k["lu_panel_f32"] > 0 and "lu_panel_f64" not in k, k
    # second-kind operators of condition below 100: a factor of 1e4 per sweep at least
    assert k["ir_norms"] <= 4 * (SWEEPS + 1), k


@pytest.mark.parametrize("direct", [True, False])
def test_sweep_of_one_body(mh, pctx, direct):
    body = mh.FloatingBody(mh.vertical_cylinder_mesh(1.0, 1.0, 40, 15, 5), ["Heave", "Surge"], body_name="c")
    p = {"wave_frequencies": np.linspace(0.5, 2.4, 5), "radiating_dofs": ["Heave", "Surge"],
         "influenced_dofs": ["Heave", "Surge"], "wave_directions": [0.3]}
    F = (mh.DirectBEM if direct else mh.IndirectBEM)(precision="mixed")
    _, k = _kernels(pctx, lambda: mh.hydrodynamic_coefficients(body, p, F, ctx=pctx))
    assert k["lu_panel_f32"] > 0 and "lu_panel_f64" not in k and k["ir_norms"] <= SWEEPS + 1, k
