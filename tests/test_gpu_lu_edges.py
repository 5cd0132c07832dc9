"""The dense LU at the sizes where its kernels change shape: panels of 1 to 16 CTAs and their
32-row chunks, ragged last panels, the tile choice of the FP64 update, in every precision."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

EPS = 2.0 ** -53


def _solve_ok(mh, ctx, n, rhs, precision, adjoint=False, scale=False):
    rng = np.random.default_rng(1000 * n + rhs)
    A = rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n))
    if scale:  # rows of very different size, so that the pivot search decides every column
        A *= 10.0 ** rng.uniform(-6, 6, n)[:, None]
    b = rng.standard_normal((n, rhs)) + 1j * rng.standard_normal((n, rhs))
    x = (mh.linsolve_adjoint if adjoint else mh.linsolve)(A, b, precision=precision, ctx=ctx)
    M = A.conj().T if adjoint else A
    # normwise backward error of Gaussian elimination with partial pivoting: a modest multiple
    # of n eps (the growth of random matrices is of order n^(2/3))
    r = np.abs(b - M @ x).max(axis=0)
    bound = 20 * n * EPS * (np.abs(M).sum(axis=1).max() * np.abs(x).max(axis=0) + np.abs(b).max(axis=0))
    assert (r <= bound).all(), (n, precision, (r / bound).max())


SIZES = [1, 2, 15, 16, 17, 31, 32, 33, 48, 63, 64, 65, 97, 129, 200, 255, 257, 415, 429, 431, 513, 700, 861]


@pytest.mark.parametrize("precision", ["fp64", "mixed", "fp64_tc"])
@pytest.mark.parametrize("n", SIZES)
def test_linsolve_sizes(mh, ctx, n, precision):
    _solve_ok(mh, ctx, n, 3, precision)


@pytest.mark.parametrize("precision", ["fp64", "fp64_tc"])
@pytest.mark.parametrize("n", [33, 200, 431])
def test_linsolve_pivoting(mh, ctx, n, precision):
    _solve_ok(mh, ctx, n, 2, precision, scale=True)


@pytest.mark.parametrize("precision", ["fp64", "mixed", "fp64_tc"])
@pytest.mark.parametrize("n", [33, 97, 431])
def test_linsolve_adjoint_sizes(mh, ctx, n, precision):
    _solve_ok(mh, ctx, n, 2, precision, adjoint=True)


@pytest.mark.parametrize("n", [40, 65])
def test_zero_column_is_reported(mh, ctx, n):
    rng = np.random.default_rng(n)
    A = rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n))
    A[:, n // 2] = 0.0
    for precision in ("fp64", "fp64_tc"):
        with pytest.raises(np.linalg.LinAlgError):
            mh.linsolve(A, np.ones(n, complex), precision=precision, ctx=ctx)


@pytest.mark.parametrize("precision", ["fp64", "mixed", "fp64_tc"])
@pytest.mark.parametrize("n, rhs", [(33, 1), (64, 9), (200, 2), (300, 17), (545, 8), (1000, 33), (1537, 5), (2999, 3)])
def test_substitution_shapes(mh, ctx, n, rhs, precision):
    # cluster sizes 1 to 16 and groups of 1 to 8 right-hand sides, whole and ragged
    _solve_ok(mh, ctx, n, rhs, precision)
    _solve_ok(mh, ctx, n, rhs, precision, adjoint=True)


@pytest.mark.parametrize("precision", ["fp64", "fp64_tc"])
@pytest.mark.parametrize("decades", [4, 8, 11])
def test_ill_conditioned_backward_error(mh, ctx, precision, decades):
    # singular values spread over `decades`: the inverted diagonal blocks keep the residual at
    # the size elimination itself leaves
    n = 320
    rng = np.random.default_rng(decades)
    q = [np.linalg.qr(rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n)))[0] for _ in range(2)]
    A = (q[0] * np.logspace(0, -decades, n)) @ q[1]
    b = rng.standard_normal((n, 2)) + 1j * rng.standard_normal((n, 2))
    x = mh.linsolve(A, b, precision=precision, ctx=ctx)
    r = np.abs(b - A @ x).max(axis=0)
    assert (r <= 20 * n * EPS * np.abs(A).sum(axis=1).max() * np.abs(x).max(axis=0)).all()


@pytest.mark.parametrize("precision", ["fp64", "mixed", "fp64_tc"])
@pytest.mark.parametrize("n", [97, 545, 1100])
def test_pivots_from_other_ctas(mh, ctx, n, precision):
    # the largest entry of column j sits n // 2 rows below (cyclically), so that every interchange
    # of the first half takes a row held by another CTA or another row block
    rng = np.random.default_rng(n)
    A = 0.3 * (rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n))) / np.sqrt(n)
    A[(np.arange(n) + n // 2) % n, np.arange(n)] += 2.0 - 1.0j
    b = rng.standard_normal((n, 2)) + 1j * rng.standard_normal((n, 2))
    x = mh.linsolve(A, b, precision=precision, ctx=ctx)
    r = np.abs(b - A @ x).max(axis=0)
    assert (r <= 20 * n * EPS * (np.abs(A).sum(axis=1).max() * np.abs(x).max(axis=0) + np.abs(b).max(axis=0))).all()


@pytest.mark.parametrize("n", [2900, 3001])
def test_two_panels_per_update(mh, ctx, n):
    # orders whose first trailing blocks have 8e6 entries or more: two FP32 panels per update, then one
    # per update, whole and ragged tiles; with a residual of n^2 products, checked as above
    rng = np.random.default_rng(n)
    A = (rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n))) / np.sqrt(n)
    A[np.arange(n), np.arange(n)] += 1.5
    b = rng.standard_normal((n, 1)) + 1j * rng.standard_normal((n, 1))
    x = mh.linsolve(A, b, precision="mixed", ctx=ctx)
    r = np.abs(b - A @ x).max(axis=0)
    assert (r <= 20 * n * EPS * (np.abs(A).sum(axis=1).max() * np.abs(x).max(axis=0) + np.abs(b).max(axis=0))).all()


@pytest.mark.parametrize("n", [40, 200, 545, 1100, 2050])
def test_refinement_settles_in_a_few_sweeps(mh, ctx, n):
    # the tensor-core residual over split and ragged column blocks: were it off in a few rows, the
    # refinement would go on to its 30th sweep (and the FP64 factorization hide it)
    rng = np.random.default_rng(n)
    A = (rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n))) / np.sqrt(n)
    A[np.arange(n), np.arange(n)] += 3.0
    b = rng.standard_normal((n, 5)) + 1j * rng.standard_normal((n, 5))
    mh.linsolve(A, b, precision="mixed", ctx=ctx)
    before = ctx.launch_count()
    x = mh.linsolve(A, b, precision="mixed", ctx=ctx)
    # five launches per panel, eight sweeps of at most seven launches, a dozen around them
    assert ctx.launch_count() - before <= 5 * ((n + 31) // 32) + 8 * 7 + 12
    r = np.abs(b - A @ x).max(axis=0)
    # the stopping rule sqrt(n) eps |A| |x| and the rounding of this check's own product
    assert (r <= (2 * np.sqrt(n) + n) * 2 * EPS * np.abs(A).sum(axis=1).max() * np.abs(x).max(axis=0)).all()


@pytest.mark.parametrize("n", [1, 31, 33, 65, 200, 450, 1041])
@pytest.mark.parametrize("rhs", [1, 8, 9])
def test_fp64_residual_products(mh, ctx, n, rhs):
    # A x and A^H x on the FP64 pipe: the adjoint solve's refinement uses them at every order
    _solve_ok(mh, ctx, n, rhs, "mixed", adjoint=True)


@pytest.mark.parametrize("precision", ["fp64", "mixed", "fp64_tc"])
@pytest.mark.parametrize("n", [1, 8, 40, 300, 1100])
@pytest.mark.parametrize("adjoint", [False, True])
def test_nan_matrix_is_refused(mh, ctx, n, precision, adjoint):
    # a NaN in the pivot search has the status of a zero pivot
    rng = np.random.default_rng(n)
    b = rng.standard_normal((n, 2)) + 0j
    for row, col in {(0, 0), (n // 2, n // 3), (n - 1, n - 1)}:
        A = rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n))
        A[row, col] = np.nan
        with pytest.raises(np.linalg.LinAlgError):
            (mh.linsolve_adjoint if adjoint else mh.linsolve)(A, b, precision=precision, ctx=ctx)


@pytest.mark.parametrize("precision", ["fp64", "fp64_tc"])
@pytest.mark.parametrize("value", [np.inf, -np.inf, complex(np.inf, np.inf), complex(1, np.inf)])
def test_infinite_matrix_is_refused(mh, ctx, precision, value):
    for n in (8, 40, 300):
        rng = np.random.default_rng(n)
        A = rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n))
        A[3, 5] = value
        with pytest.raises(np.linalg.LinAlgError):
            mh.linsolve(A, rng.standard_normal((n, 2)) + 0j, precision=precision, ctx=ctx)


@pytest.mark.parametrize("bits", [23, 24, 25, 31, 40, 52, 53])
@pytest.mark.parametrize("unit", [1.0, -1.0, 1j, -1j])
def test_entries_just_below_a_power_of_two(mh, ctx, bits, unit):
    # multipliers and rows of U just below one, the largest fixed-point numbers of the exact digits:
    # symmetric meshes have such multipliers
    n = 200
    rng = np.random.default_rng(bits)
    A = 0.2 * (rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n))) / np.sqrt(n) + 2.0 * np.eye(n)
    near = 1.0 - 2.0 ** -bits
    A[0, 0] = 1.0
    A[40:80, 0] = unit * near
    A[0, 100:140] = near
    A[64, 64] = 4.0
    A[150:160, 64] = 4.0 * unit * near
    b = rng.standard_normal((n, 2)) + 0j
    x = mh.linsolve(A, b, precision="fp64_tc", ctx=ctx)
    r = np.abs(b - A @ x).max(axis=0)
    assert (r <= 20 * n * EPS * (np.abs(A).sum(axis=1).max() * np.abs(x).max(axis=0) + np.abs(b).max(axis=0))).all()
