"""More pieces of large triangles than 32 bits count: 26845 copies of one sliver that crosses all 5000 x 4096
columns of a grid, 160000 pieces each.  The copies lie above the grid, so no voxel is a boundary voxel
and an odd number of them has the parity of one; the list has room for one of them, and the rest stay
with their groups."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_more_pieces_than_32_bits(built):
    import torch

    gpv = built
    one = np.array([0, 0, 2, 1, 1, 2.5, 0.5, 0.501, 2.2], np.float32)
    spec = gpv.GridSpec()
    spec.bbox_min[:], spec.bbox_max[:], spec.ndiv[:], spec.ndiv2[:] = [0.0] * 3, [1.0] * 3, [5000, 4096, 1], [0] * 3
    ctx = gpv.Context(0)
    try:
        states = []
        for copies in (1, 2, 26845):
            assert copies < 3 or copies * (5000 * 4096 // 32 // 4) > 1 << 32
            d = torch.from_numpy(np.tile(one, copies)).cuda()
            res = ctx.voxelize_device(d.data_ptr(), copies, spec)
            states.append(ctx.fetch(res)[0])
            assert res.num_boundary == 0
            ctx.release(res)
        assert (states[0] == 127).sum() > 4096 and not states[1].any()
        np.testing.assert_array_equal(states[2], states[0])
    finally:
        ctx.close()
