"""Calls whose (voxel, triangle) records do not fit their buffer: records collected by a warp and records
of tall columns that go straight to the buffer, with capacities that none, some and nearly all of them
exceed.  The call runs again with the exact capacity, once, and equals the oracle."""
import numpy as np
import pytest

from oracle import oracle as orc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [(6, 5, 700), (40, 41, 42)])
@pytest.mark.parametrize("capacity", [1, 127, 5000, "all but one"])
def test_records_past_the_capacity(built, n, capacity):
    gpv = built
    tris = gpv.gen_torus(9, 40, 20, (0.5, 0.5, 0.5), 0.35, 0.12, 0.004)
    spec = gpv.grid_padded(*gpv.mesh_bounds(tris), n, (3, 2, 2))
    ref = orc.Run(tris, spec, fill=orc.FILL_CAND)
    pairs = int(ref.L.orc_num_pairs(ref.h))
    assert pairs > 5000
    for batch in (False, True):
        ctx = gpv.Context(0)
        try:
            ctx.set_debug("pair_capacity", pairs - 1 if capacity == "all but one" else capacity)
            if batch:
                import torch

                other = gpv.gen_uvsphere(4, 24, 12, (0.5, 0.5, 0.5), 0.3, 0.002)
                sp2 = gpv.grid_padded(*gpv.mesh_bounds(other), 12, 2)
                ref2 = orc.Run(other, sp2, fill=orc.FILL_CAND)
                d = [torch.from_numpy(t).cuda() for t in (other, tris, other)]
                torch.cuda.synchronize()
                res = ctx.voxelize_batch([x.data_ptr() for x in d], [x.numel() // 9 for x in d], [sp2, spec, sp2])
                want = [ref2, ref, ref2]
            else:
                res, want = [ctx.voxelize_host(tris, spec)], [ref]
            assert ctx.get_debug("replans") == 1
            for r, w in zip(res, want):
                l1, pre, bi, l2 = ctx.fetch(r)
                np.testing.assert_array_equal(l1, w.level1_bytes())
                np.testing.assert_array_equal(pre, w.prefix())
                np.testing.assert_array_equal(bi, w.boundary_index())
                np.testing.assert_array_equal(l2, w.level2_bytes())
                ctx.release(r)
        finally:
            ctx.close()
