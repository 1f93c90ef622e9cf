"""SAT runs of grids near to and far from the origin in one call: far from it a run has only a few pairs.
Every mesh's states equal the oracle's, alone and in the batch."""
import numpy as np
import pytest

from oracle import oracle as orc

pytestmark = pytest.mark.gpu


def test_batch_of_near_and_far_grids(ctx, built):
    gpv = built
    torch = pytest.importorskip("torch")

    meshes, specs = [], []
    for k, (offset, n, n2) in enumerate([(0.0, (24, 20, 18), 4), (10000.0, (22, 25, 19), 8), (0.0, 3, 6),
                                         (2000.0, (31, 17, 26), (3, 5, 16)), (-40000.0, 12, 9), (0.0, (30, 9, 33), 5)]):
        t = gpv.gen_torus(k, 40, 20, (0.5, 0.5, 0.5), 0.35, 0.12, 0.004) + np.float32(offset)
        meshes.append(np.ascontiguousarray(t, np.float32))
        specs.append(gpv.grid_padded(*gpv.mesh_bounds(meshes[-1]), n, n2))
    dev = [torch.from_numpy(t).cuda() for t in meshes]
    batch = ctx.voxelize_batch([d.data_ptr() for d in dev], [t.size // 9 for t in meshes], specs)
    for t, s, r in zip(meshes, specs, batch):
        ref = orc.Run(t, s, fill=orc.FILL_CAND)
        alone = ctx.voxelize_host(t, s)
        for res in (r, alone):
            l1, _, bi, l2 = ctx.fetch(res)
            np.testing.assert_array_equal(l1, ref.level1_bytes())
            np.testing.assert_array_equal(bi, ref.boundary_index())
            np.testing.assert_array_equal(l2, ref.level2_bytes())
            ctx.release(res)
