"""The Birk Rankine assembly (far terms per thread, near terms from a list) at ragged row and
column tiles, both formulations, image signs and the no-allocation entry point's in-place static
part, against the oracle."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

KINDS = {"direct_only": (1, 0), "image": (1, 2), "negative": (1, 4), "image_only": (0, 2)}


@pytest.mark.parametrize("n_lat, n_lon", [(1, 3), (3, 5), (7, 18), (8, 16), (9, 15), (16, 41)])
@pytest.mark.parametrize("kinds", list(KINDS))
@pytest.mark.parametrize("direct", [True, False])
def test_static_tiles(mh, oracle, ctx, n_lat, n_lon, kinds, direct):
    mesh = mh.hemisphere_mesh(1.3, n_lat, n_lon)
    gfs = sum(KINDS[kinds])
    names = {1: mh.Rankine, 2: mh.RankineReflected, 4: mh.RankineReflectedNegative}
    S, D = mh.assemble_matrices(tuple(names[b]() for b in (1, 2, 4) if gfs & b), mesh, 1.0, direct=direct, ctx=ctx)
    So, Do = oracle.assemble_matrices(mesh, 1.0, gfs=gfs, direct=direct)
    # entries differ by a few roundings of the terms they sum (at most 2 pi and 1/r^2 of them)
    assert np.abs(S - So).max() <= 64 * 2.0 ** -53 * np.abs(So).max()
    assert np.abs(D - Do).max() <= 64 * 2.0 ** -53 * max(1.0, np.abs(Do).max())


@pytest.mark.parametrize("n_lat, n_lon", [(1, 3), (8, 16), (16, 41)])
@pytest.mark.parametrize("direct", [True, False])
@pytest.mark.parametrize("fixed", [None, (1.0, 0.0, 0.0)])
def test_noalloc_equals_allocating(mh, ctx, n_lat, n_lon, direct, fixed):
    torch = pytest.importorskip("torch")
    mesh = mh.hemisphere_mesh(1.3, n_lat, n_lon)
    n, L = mesh.nfaces, mh.load_library()
    dev = [torch.from_numpy(np.ascontiguousarray(a, dtype=np.float64)).cuda()
           for a in (mesh.panel_vertices, mesh.centers, mesh.normals, mesh.areas, mesh.radii)]
    for greens in ((mh.Rankine(), mh.RankineReflected(), mh.GFWu()), (mh.Rankine(),), (mh.GFWu(),)):
        S = torch.full((n, n), float("nan"), dtype=torch.complex128, device="cuda")
        D = torch.full_like(S, float("nan"))
        fx = None if fixed is None else np.asarray(fixed)
        rc = L.mh_assemble_matrices_noalloc(torch.cuda.current_stream().cuda_stream, n, *[t.data_ptr() for t in dev],
                                            0.8, mh.gf_flags(greens), int(direct), 1,
                                            None if fx is None else fx.ctypes.data_as(ctypes.c_void_p), S.data_ptr(),
                                            D.data_ptr())
        assert rc == 0
        torch.cuda.synchronize()
        S0, D0 = mh.assemble_matrices(greens, mesh, 0.8, direct=direct, all_normals=fixed, ctx=ctx)
        assert np.array_equal(S.cpu().numpy().T, S0) and np.array_equal(D.cpu().numpy().T, D0)


@pytest.mark.parametrize("field, entry", [("centers", (5, 0)), ("centers", (5, 2)), ("panel_vertices", (5, 1, 1))])
@pytest.mark.parametrize("gfs", [1, 3, 5, 35])
@pytest.mark.parametrize("direct", [True, False])
def test_nan_geometry_stays_nan(mh, field, entry, gfs, direct):
    # device buffers are not checked for NaN (host meshes are): what a NaN enters has to come out as
    # NaN, never as a number
    torch = pytest.importorskip("torch")
    mesh = mh.hemisphere_mesh(1.0, 6, 12)
    n, L = mesh.nfaces, mh.load_library()
    arrays = {f: np.array(getattr(mesh, f), dtype=np.float64)
              for f in ("panel_vertices", "centers", "normals", "areas", "radii")}
    arrays[field][entry] = np.nan
    dev = [torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in arrays.values()]
    S = torch.zeros((n, n), dtype=torch.complex128, device="cuda")
    D = torch.zeros_like(S)
    rc = L.mh_assemble_matrices_noalloc(torch.cuda.current_stream().cuda_stream, n, *[t.data_ptr() for t in dev], 0.8,
                                        gfs, int(direct), 1, None, S.data_ptr(), D.data_ptr())
    assert rc == 0
    torch.cuda.synchronize()
    S, D = S.cpu().numpy().T, D.cpu().numpy().T
    # panel 5 as the source: the near integral takes its corners, the wave term its centre; as the
    # field point: every term takes its centre
    if field == "panel_vertices" or gfs & 32:
        assert np.isnan(S[:, 5]).all() and np.isnan(D[:, 5]).all()
    if field == "centers":
        assert np.isnan(S[5]).all() and np.isnan(D[5]).all()
    keep = np.arange(n) != 5
    assert np.isfinite(S[np.ix_(keep, keep)]).all() and np.isfinite(D[np.ix_(keep, keep)]).all()
