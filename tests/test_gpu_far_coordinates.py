"""Meshes far from the origin, up to several Level2 cells to a float: the centre tables leave their affine
form, neighbouring ray origins can round to one height, and most cells run the exact tests.  Every state
equals the oracle's."""
import numpy as np
import pytest

from oracle import oracle as orc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("offset", [30.0, 1000.0, -3000.0, 10000.0, 50000.0])
@pytest.mark.parametrize("n2", [(8, 8, 8), (5, 4, 7), (16, 16, 16), (1, 2, 32)])
def test_states(ctx, built, offset, n2):
    gpv = built
    tris = gpv.gen_torus(21, 48, 24, (0.5, 0.5, 0.5), 0.35, 0.12, 0.004)
    shift = np.array([offset, 0.7 * offset, -1.3 * offset], np.float32)
    tris = np.ascontiguousarray((tris.reshape(-1, 3) + shift).astype(np.float32)).reshape(-1)
    spec = gpv.grid_padded(*gpv.mesh_bounds(tris), (30, 27, 12), n2)
    ref = orc.Run(tris, spec, fill=orc.FILL_CAND)
    res = ctx.voxelize_host(tris, spec)
    l1, pre, bi, l2 = ctx.fetch(res)
    assert ref.B > 500
    np.testing.assert_array_equal(l1, ref.level1_bytes())
    np.testing.assert_array_equal(pre, ref.prefix())
    np.testing.assert_array_equal(bi, ref.boundary_index())
    np.testing.assert_array_equal(l2, ref.level2_bytes())
    ctx.release(res)


@pytest.mark.parametrize("offset", [3000.0, 10000.0])
def test_few_voxels_share_their_pairs(ctx, built, offset):
    gpv = built
    tris = gpv.gen_uvsphere(5, 64, 32, (0.5, 0.5, 0.5), 0.4, 0.002)
    tris = np.ascontiguousarray((tris + np.float32(offset)).astype(np.float32))
    spec = gpv.grid_padded(*gpv.mesh_bounds(tris), 5, 8)
    ref = orc.Run(tris, spec, fill=orc.FILL_CAND)
    res = ctx.voxelize_host(tris, spec)
    l1, _, bi, l2 = ctx.fetch(res)
    np.testing.assert_array_equal(l1, ref.level1_bytes())
    np.testing.assert_array_equal(bi, ref.boundary_index())
    np.testing.assert_array_equal(l2, ref.level2_bytes())
    ctx.release(res)
