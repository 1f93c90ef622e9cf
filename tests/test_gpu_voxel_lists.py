"""Lists of a voxel's triangles at the lengths where their handling changes: the counting sort with each
list ordered in registers, in a warp's or a block's shared memory or in place, and the radix sort for
long averages; Level1 sums by a thread or a warp; Level2 sums in tiles; and SAT items shared by several
warps.  Normals are float sums in list order, so every value equals the oracle's."""
import numpy as np
import pytest

from oracle import oracle as orc

pytestmark = pytest.mark.gpu


def _cluster(n, at, size, seed):
    rng = np.random.default_rng(seed)
    c = np.asarray(at) + rng.uniform(-size, size, (n, 1, 3))
    return c + rng.normal(size=(n, 3, 3)) * size * 0.3


def _check(ctx, gpv, tris, spec):
    tris = np.ascontiguousarray(tris, np.float32).reshape(-1)
    ref = orc.Run(tris, spec, fill=orc.FILL_CAND)
    ctx.set_normals(gpv.NORMALS_FLOAT)
    try:
        res = ctx.voxelize_host(tris, spec)
        l1, pre, bi, l2 = ctx.fetch(res)
        n1, n2 = ctx.fetch_normals(res)
        ctx.release(res)
    finally:
        ctx.set_normals(gpv.NORMALS_OFF)
    np.testing.assert_array_equal(l1, ref.level1_bytes())
    np.testing.assert_array_equal(bi, ref.boundary_index())
    np.testing.assert_array_equal(l2, ref.level2_bytes())
    np.testing.assert_array_equal(n1, ref.level1_normals())
    np.testing.assert_array_equal(n2, ref.level2_normals())


@pytest.mark.parametrize("heap,n2", [(20, (3, 3, 3)), (70, (8, 8, 8)), (600, (5, 4, 3)), (3000, (2, 2, 2)),
                                     (9000, (4, 4, 4))])
def test_one_long_list_among_short_ones(ctx, built, heap, n2):
    # a sphere's short lists and a heap of small triangles within one voxel
    gpv = built
    s = gpv.gen_uvsphere(3, 300, 150, (0, 0, 0), 0.45, 0.001).reshape(-1, 3, 3)
    tris = np.concatenate([s, _cluster(heap, (0.011, 0.013, 0.017), 0.002, heap)])
    _check(ctx, gpv, tris, gpv.grid_padded((-0.46,) * 3, (0.46,) * 3, (25, 24, 27), n2))


@pytest.mark.parametrize("n1,n2", [((3, 3, 3), (4, 4, 4)), ((4, 5, 3), (16, 16, 16)), ((8, 8, 8), (7, 5, 3)),
                                   ((3, 4, 3), (32, 16, 3))])
def test_few_voxels_with_long_lists(ctx, built, n1, n2):
    gpv = built
    tris = gpv.gen_torus(8, 60, 40, (0, 0, 0), 0.35, 0.12, 0.01)
    mn, mx = gpv.mesh_bounds(tris)
    _check(ctx, gpv, tris, gpv.grid_padded(mn, mx, n1, n2))
