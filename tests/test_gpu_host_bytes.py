"""Level2 states written into page-locked host memory for layouts without the 16-cell groups: voxels around
the size from which they go out 16 bytes at a time, single layers and columns, blocks that start at every
offset from a 16-byte boundary, both fills.  Bytes, counts and what lies past the output equal the
device-resident call's and are untouched."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n2", [(1, 1, 1), (3, 3, 3), (7, 3, 3), (4, 4, 4), (5, 13, 1), (1, 1, 32), (1, 32, 3), (32, 32, 1),
                                (5, 5, 5), (3, 3, 8), (6, 5, 16), (15, 15, 15), (31, 7, 17), (32, 32, 32)])
@pytest.mark.parametrize("fill", ["ray", "stencil"])
def test_other_layouts(built, n2, fill):
    import torch

    gpv = built
    tris = gpv.gen_torus(17, 48, 24, (0.5, 0.5, 0.5), 0.35, 0.12, 0.004)
    spec = gpv.grid_padded(*gpv.mesh_bounds(tris), (19, 17, 14), n2)
    ctx = gpv.Context(0)
    try:
        ctx.set_fill(gpv.FILL_STENCIL if fill == "stencil" else gpv.FILL_RAY)
        want = ctx.voxelize_host(tris, spec)
        w = ctx.fetch(want)
        n1, b, size = want.num_level1, want.num_boundary, w[3].size
        t = torch.from_numpy(tris).pin_memory()
        l1 = torch.empty(n1, dtype=torch.uint8, pin_memory=True)
        pre = torch.empty(n1, dtype=torch.int32, pin_memory=True)
        idx = torch.empty(b, dtype=torch.int32, pin_memory=True)
        l2 = torch.full((size + 64,), 0xA5, dtype=torch.uint8).pin_memory()
        for _ in range(2):
            l2.fill_(0xA5)
            rc, r = ctx.voxelize_to_host(t.data_ptr(), tris.size // 9, spec, l1.data_ptr(), pre.data_ptr(), idx.data_ptr(),
                                         l2.data_ptr(), size)
            assert rc == 0
            for got, exp in zip((l1, pre, idx, l2[:size]), w):
                np.testing.assert_array_equal(got.numpy(), exp)
            assert (l2[size:] == 0xA5).all()
            assert (r.num_level2_inside, r.num_level2_boundary) == (want.num_level2_inside, want.num_level2_boundary)
            ctx.release(r)
        ctx.release(want)
    finally:
        ctx.close()
