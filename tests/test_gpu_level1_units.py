"""The Level1 kernel's units against the oracle where their split and their bounds can go wrong: one
triangle to a few per group (shared by several warps), triangles over the whole grid (the list of
pieces), z runs cut to the triangle's plane, columns of one layer to several words, near-vertical and
sliver triangles (no bound on the ray's height), meshes far from the origin, and the allocation-free
entry on the same engine.  States and counts are decisions, so every one is equal."""
import ctypes as C

import numpy as np
import pytest

from oracle import oracle as orc

pytestmark = pytest.mark.gpu


def _box(q):
    c = np.array([[x, y, z] for x in (0, 1) for y in (0, 1) for z in (0, 1)], np.float64) - 0.5
    f = [(0, 1, 3), (0, 3, 2), (4, 6, 7), (4, 7, 5), (0, 4, 5), (0, 5, 1), (2, 3, 7), (2, 7, 6), (0, 2, 6), (0, 6, 4),
         (1, 5, 7), (1, 7, 3)]
    return (c @ q.T)[np.array(f)]


def _mesh(name, gpv):
    rng = np.random.default_rng(11)
    q, _ = np.linalg.qr(rng.normal(size=(3, 3)))
    if name == "box":
        return _box(q)
    if name == "upright":  # near-vertical walls: tiny x/y projections
        a = 2e-6
        return _box(np.array([[1, 0, a], [0, 1, a], [-a, -a, 1.0]]))
    if name == "slivers":
        t = rng.uniform(-0.5, 0.5, (40, 3, 3))
        t[:, 2] = t[:, 1] + rng.normal(size=(40, 3)) * 10.0 ** rng.uniform(-7, -2, (40, 1))
        return np.concatenate([_box(q), t])
    if name == "one":
        return rng.uniform(-0.5, 0.5, (1, 3, 3))
    if name == "mixed":  # two triangles over the grid among many small ones
        s = gpv.gen_uvsphere(3, 40, 20, (0, 0, 0), 0.45, 0.01).reshape(-1, 3, 3)
        return np.concatenate([s[:300], rng.uniform(-0.5, 0.5, (2, 3, 3)), s[300:]])
    return gpv.gen_torus(4, 60, 30, (0.0, 0.0, 0.0), 0.35, 0.12, 0.01).reshape(-1, 3, 3)


def _noalloc(gpv, tris, spec):
    torch = pytest.importorskip("torch")
    n1 = int(np.prod(list(spec.ndiv)))
    t = torch.from_numpy(tris).cuda()
    l1 = torch.zeros(n1, dtype=torch.uint8, device="cuda")
    pre = torch.zeros(n1, dtype=torch.int32, device="cuda")
    bi = torch.zeros(n1, dtype=torch.int32, device="cuda")
    b = C.c_int64()
    rc = gpv.lib().gpv_voxelize_level1_noalloc(t.data_ptr(), tris.size // 9, C.byref(spec), l1.data_ptr(),
                                               pre.data_ptr(), bi.data_ptr(), C.byref(b), None)
    assert rc == 0, gpv.lib().gpv_noalloc_last_error()
    return l1.cpu().numpy(), pre.cpu().numpy(), bi.cpu().numpy()[:b.value]


@pytest.mark.parametrize("mesh", ["box", "upright", "slivers", "one", "mixed", "torus"])
@pytest.mark.parametrize("n1", [(65, 33, 97), (40, 37, 3), (6, 5, 200), (96, 96, 64)])
def test_level1_units(ctx, built, mesh, n1):
    gpv = built
    tris = np.ascontiguousarray(_mesh(mesh, gpv), np.float32).reshape(-1)
    mn, mx = gpv.mesh_bounds(tris)
    for shift in ((0, 0, 0), (300.0, -2000.0, 5000.0)) if n1[0] == 40 else ((0, 0, 0),):
        t = np.ascontiguousarray(tris.reshape(-1, 3) + np.asarray(shift, np.float32), np.float32).reshape(-1)
        mn, mx = gpv.mesh_bounds(t)
        for n2 in (0, 1):
            spec = gpv.grid_padded(mn, mx, n1, n2)
            ref = orc.Run(t, spec, fill=orc.FILL_CAND)
            res = ctx.voxelize_host(t, spec)
            l1, pre, bi, _ = ctx.fetch(res)
            np.testing.assert_array_equal(l1, ref.level1_bytes())
            np.testing.assert_array_equal(pre, ref.prefix())
            np.testing.assert_array_equal(bi, ref.boundary_index())
            assert res.num_pairs == ref.num_pairs()
            assert (res.work.sat1, res.work.ray1) == (ref.sat1_tests(), ref.ray1_candidates())
            ctx.release(res)
        l1n, pren, bin_ = _noalloc(gpv, t, spec)
        np.testing.assert_array_equal(l1n, l1)
        np.testing.assert_array_equal(pren, pre)
        np.testing.assert_array_equal(bin_, bi)
