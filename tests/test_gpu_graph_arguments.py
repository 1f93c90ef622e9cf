"""A recorded graph is replayed only for calls with the same launch arguments: a call that adds a Level2
grid of one cell to a grid so small that every buffer keeps its place (the marks plane exists only with
Level2), and batches whose meshes swap their sub-grids, which keeps every count but the size of the SAT
masks.  Every call equals the oracle."""
import numpy as np
import pytest

from oracle import oracle as orc

pytestmark = pytest.mark.gpu


def _equal(ctx, res, tris, spec):
    ref = orc.Run(tris, spec, fill=orc.FILL_CAND)
    l1, pre, bi, l2 = ctx.fetch(res)
    np.testing.assert_array_equal(l1, ref.level1_bytes())
    np.testing.assert_array_equal(pre, ref.prefix())
    np.testing.assert_array_equal(bi, ref.boundary_index())
    if spec.ndiv2[0]:
        np.testing.assert_array_equal(l2, ref.level2_bytes())


@pytest.mark.parametrize("graphs", ["two", "one"])
@pytest.mark.parametrize("n", [(3, 3, 3), (4, 4, 4), (31, 4, 8), (5, 6, 5)])
def test_level2_of_one_cell_after_level1(built, n, graphs):
    import torch

    gpv = built
    tris = gpv.gen_uvsphere(3, 24, 12, (0.5, 0.5, 0.5), 0.4, 0.002)
    spec = {k: gpv.grid_padded(*gpv.mesh_bounds(tris), n, (k, k, k)) for k in (0, 1)}
    d = torch.from_numpy(tris).cuda()
    torch.cuda.synchronize()
    ctx, stream = gpv.Context(0), torch.cuda.Stream()  # (the default stream takes no recording)
    try:
        ctx.set_graphs(ctx.GRAPHS_TWO if graphs == "two" else ctx.GRAPHS_ONE)
        for k in (0, 0, 0, 1, 1, 0, 1, 0, 0, 1):
            res = ctx.voxelize_device(d.data_ptr(), tris.size // 9, spec[k], stream.cuda_stream)
            _equal(ctx, res, tris, spec[k])
            ctx.release(res)
    finally:
        ctx.close()


@pytest.mark.parametrize("mode", ["normals", "stencil"])
def test_swapped_sub_grids(built, mode):
    import torch

    gpv = built
    # few voxels (their SAT pairs are shared by warps into cleared masks), a small and a large mesh
    small = gpv.gen_uvsphere(5, 32, 16, (0.5, 0.5, 0.5), 0.1, 0.002)
    large = gpv.gen_uvsphere(6, 32, 16, (0.5, 0.5, 0.5), 0.4, 0.002)
    tris = [small, large]
    dev = [torch.from_numpy(t).cuda() for t in tris]
    lo, hi = (0.0, 0.0, 0.0), (1.0, 1.0, 1.0)

    def specs(a, b):
        out = []
        for n2 in (a, b):
            s = gpv.GridSpec()
            s.bbox_min[:], s.bbox_max[:], s.ndiv[:], s.ndiv2[:] = lo, hi, [6, 6, 6], [n2] * 3
            out.append(s)
        return out

    ctx, stream = gpv.Context(0), torch.cuda.Stream()
    torch.cuda.synchronize()
    try:
        if mode == "normals":
            ctx.set_normals(gpv.NORMALS_FLOAT)
        else:
            ctx.set_fill(gpv.FILL_STENCIL)
        big = specs(8, 8)
        for a, b in ((8, 2), (2, 8), (8, 2), (8, 2), (2, 8), (2, 8)):
            # masks of other voxels where the next calls' will lie
            ctx.set_graphs(False)
            for r in ctx.voxelize_batch([dev[1].data_ptr()] * 2, [large.size // 9] * 2, big,
                                         stream.cuda_stream):
                ctx.release(r)
            ctx.set_graphs(ctx.GRAPHS_TWO)
            sp = specs(a, b)
            res = ctx.voxelize_batch([t.data_ptr() for t in dev], [t.size // 9 for t in tris], sp,
                                     stream.cuda_stream)
            for r, t, s in zip(res, tris, sp):
                ref = orc.Run(t, s, fill=orc.FILL_STENCIL if mode == "stencil" else orc.FILL_CAND)
                l1, _, bi, l2 = ctx.fetch(r)
                np.testing.assert_array_equal(l1, ref.level1_bytes())
                np.testing.assert_array_equal(bi, ref.boundary_index())
                np.testing.assert_array_equal(l2, ref.level2_bytes())
                if mode == "normals":
                    n1, n2 = ctx.fetch_normals(r)
                    np.testing.assert_array_equal(n1, ref.level1_normals())
                    np.testing.assert_array_equal(n2, ref.level2_normals())
            for r in res:
                ctx.release(r)
    finally:
        ctx.close()
