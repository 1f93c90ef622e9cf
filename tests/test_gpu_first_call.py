"""First calls on a new context whose (voxel, triangle) records exceed the first buffer (the call runs
again with a larger one): every kind of call gives the outputs of a later call, host outputs included,
and a Level1 call, whose records are only counted, leaves the buffer's size to the Level2 call after it."""
import numpy as np
import pytest

from oracle import oracle as orc

pytestmark = pytest.mark.gpu

N, N2 = (150, 140, 160), (2, 1, 2)


def _box(gpv):
    rng = np.random.default_rng(4)
    c = np.array([[x, y, z] for x in (0, 1) for y in (0, 1) for z in (0, 1)], np.float64) - 0.5
    f = [(0, 1, 3), (0, 3, 2), (4, 6, 7), (4, 7, 5), (0, 4, 5), (0, 5, 1), (2, 3, 7), (2, 7, 6), (0, 2, 6), (0, 6, 4),
         (1, 5, 7), (1, 7, 3)]
    q, _ = np.linalg.qr(rng.normal(size=(3, 3)))
    tris = np.ascontiguousarray((c @ q.T)[np.array(f)], np.float32).reshape(-1)
    mn, mx = gpv.mesh_bounds(tris)
    return tris, gpv.grid_padded(mn, mx, N, N2), gpv.grid_padded(mn, mx, N)


@pytest.mark.parametrize("level1_first", [False, True])
@pytest.mark.parametrize("kind", ["device", "to_host", "to_host_slabs", "normals", "stencil"])
def test_first_call_overflows(built, kind, level1_first):
    import torch

    gpv = built
    tris, spec, flat = _box(gpv)
    ref = orc.Run(tris, spec, fill=orc.FILL_STENCIL if kind == "stencil" else orc.FILL_CAND)
    want = ref.level1_bytes(), ref.prefix(), ref.boundary_index(), ref.level2_bytes()
    assert ref.num_pairs() > 1 << 16  # (the first buffer's records)
    ctx = gpv.Context(0)
    try:
        if level1_first:
            r = ctx.voxelize_host(tris, flat)
            ctx.release(r)
        if kind == "stencil":
            ctx.set_fill(gpv.FILL_STENCIL)
        if kind == "normals":
            ctx.set_normals(gpv.NORMALS_FLOAT)
        h = torch.from_numpy(tris).pin_memory()
        if kind.startswith("to_host"):
            out = [torch.full((w.size * w.itemsize,), 77, dtype=torch.uint8).pin_memory() for w in want]
            rc, res = ctx.voxelize_to_host(h.data_ptr(), tris.size // 9, spec, *[o.data_ptr() for o in out],
                                           want[3].size, 3 if kind.endswith("slabs") else 0)
            assert rc == 0
            got = [o.numpy().view(w.dtype) for o, w in zip(out, want)]
        else:
            res = ctx.voxelize_host(tris, spec)
            got = ctx.fetch(res)
        for g, w in zip(got, want):
            np.testing.assert_array_equal(g, w)
        if kind == "normals":
            np.testing.assert_array_equal(ctx.fetch_normals(res)[1], ref.level2_normals())
        ctx.release(res)
    finally:
        ctx.close()
