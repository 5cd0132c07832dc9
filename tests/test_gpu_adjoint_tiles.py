"""The static and wave adjoint at ragged row and column tiles (fewer panels than a tile, one row
past it, several tiles), both formulations, against central differences of the device sweep along
affine vertex moves (every panel stays planar)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

OMEGAS = (0.7, 1.6)
H = 1e-6


def _body(mh, vertices, faces):
    return mh.FloatingBody(mh.StaticArraysMesh(vertices, faces), ["Heave", "Surge"])


def _objective(mh, ctx, body, F):
    names = list(body.dofs)
    r = mh.hydrodynamic_coefficients(body, {"wave_frequencies": OMEGAS, "radiating_dofs": names,
                                            "influenced_dofs": names}, F, ctx=ctx, rho=1025.0, g=9.81)
    return sum(r[k][h, h].sum() for k in ("added_mass", "radiation_damping") for h in range(len(names)))


@pytest.mark.parametrize("shape", [(2, 1, 1), (3, 3, 2), (8, 4, 3), (12, 5, 2), (10, 6, 4)])  # 6 .. 188 panels
@pytest.mark.parametrize("direct", [True, False])
@pytest.mark.parametrize("sign", ["reflected", "negative"])
def test_gradient_along_affine_moves(mh, ctx, shape, direct, sign):
    base = mh.barge_mesh(4.0, 2.0, 1.0, *shape)
    image = mh.RankineReflected() if sign == "reflected" else mh.RankineReflectedNegative()
    F = (mh.DirectBEM if direct else mh.IndirectBEM)((mh.Rankine(), image, mh.GFWu()))
    V = base.vertices - [0.0, 0.0, 0.05]
    J, grad = mh.hydro_gradient(_body(mh, V, base.faces), OMEGAS, ["Heave", "Surge"], F, ctx=ctx, rho=1025.0, g=9.81)
    assert abs(J - _objective(mh, ctx, _body(mh, V, base.faces), F)) <= 1e-12 * abs(J)
    rng = np.random.default_rng(sum(shape))
    for _ in range(2):
        M = rng.standard_normal((3, 3))
        M[2, :2] = 0.0
        d = V @ M.T
        fd = (_objective(mh, ctx, _body(mh, V + H * d, base.faces), F)
              - _objective(mh, ctx, _body(mh, V - H * d, base.faces), F)) / (2 * H)
        ad = float(np.sum(grad * d))
        # differences at h = 1e-6 carry 1e-9 of rounding; the scale covers moves that cancel
        assert abs(ad - fd) <= 1e-6 * max(abs(fd), 1e-3 * np.abs(grad).sum() * np.abs(d).max()), (ad, fd)
