"""The stencil fill where the SAT's rounding is large against the Level2 cells: a triangle that no voxel
records from some height up can still cover samples above that voxel's first clip heights.  Every state
equals the oracle's, whatever the chunks that a column is cut into."""
import numpy as np
import pytest

from oracle import oracle as orc

pytestmark = pytest.mark.gpu


def _sheet(rng, count):
    t = rng.random((count, 1, 3)) + rng.normal(size=(count, 3, 3)) * 0.01
    t[..., 2] = t[..., 2] * 0.02 + 0.5
    return t


def _slivers(rng, count):
    a = rng.random((count, 1, 3))
    b = a + rng.normal(size=(count, 1, 3)) * 0.3
    return np.concatenate([a, b, b + rng.normal(size=(count, 1, 3)) * 0.003], 1)


@pytest.mark.parametrize("shape,count,offset,n,n2", [
    (_sheet, 1339, 10000.0, (41, 63, 63), (14, 15, 13)),  # heights that do not increase
    (_sheet, 4044, 10000.0, (35, 28, 25), (6, 6, 6)),
    (_sheet, 4692, 1000.0, (19, 20, 19), (16, 16, 16)),
    (_sheet, 4919, 10000.0, (53, 76, 82), (4, 4, 4)),
    (_slivers, 1500, 1000.0, (30, 41, 28), (5, 7, 6)),
    (_slivers, 1500, 0.0, (30, 41, 28), (5, 7, 6)),
])
@pytest.mark.parametrize("cap", [1, 3, 16, 32])
def test_states(ctx, built, shape, count, offset, n, n2, cap):
    gpv = built
    tris = (shape(np.random.default_rng(count), count) + offset).astype(np.float32).reshape(-1)
    spec = gpv.grid_padded(*gpv.mesh_bounds(tris), n, n2)
    ref = orc.Run(tris, spec, fill=orc.FILL_STENCIL)
    ctx.set_fill(gpv.FILL_STENCIL)
    ctx.set_level2_chunk(cap)
    try:
        res = ctx.voxelize_host(tris, spec)
    finally:
        ctx.set_fill(gpv.FILL_RAY)
        ctx.set_level2_chunk(16)
    l1, _, bi, l2 = ctx.fetch(res)
    ctx.release(res)
    assert ref.B > 200
    np.testing.assert_array_equal(l1, ref.level1_bytes())
    np.testing.assert_array_equal(bi, ref.boundary_index())
    np.testing.assert_array_equal(l2, ref.level2_bytes())
