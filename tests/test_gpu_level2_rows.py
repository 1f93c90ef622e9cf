"""The row-solved Level2 SAT and fill against the oracle where their intervals, batches and error
bounds can go wrong: one sub-cell to 32 per axis, uneven sub-grids whose columns straddle mask words,
more rows than one batch holds, triangles far larger than a voxel, meshes far from the origin (every
cell uncertain), and coordinates outside the magnitudes the bounds are used for (exact tests only).
States are decisions, so every byte and count is equal."""
import numpy as np
import pytest

from oracle import oracle as orc

pytestmark = pytest.mark.gpu


def _spec(gpv, mn, mx, n, n2):
    s = gpv.GridSpec()
    s.bbox_min[:] = [float(v) for v in mn]
    s.bbox_max[:] = [float(v) for v in mx]
    s.ndiv[:] = n
    s.ndiv2[:] = n2
    return s


def _check(ctx, gpv, tris, spec):
    ref = orc.Run(tris, spec, fill=orc.FILL_CAND)
    for _ in range(3):  # two phases, then one graph
        res = ctx.voxelize_host(tris, spec)
        l1, pre, bi, l2 = ctx.fetch(res)
        np.testing.assert_array_equal(l1, ref.level1_bytes())
        np.testing.assert_array_equal(bi, ref.boundary_index())
        np.testing.assert_array_equal(l2, ref.level2_bytes())
        assert res.num_level2_boundary == int((l2 == 254).sum())
        assert res.num_level2_inside == int((l2 == 127).sum())
        ctx.release(res)


@pytest.mark.parametrize("n2", [(1, 1, 1), (2, 1, 3), (5, 5, 5), (7, 3, 13), (8, 8, 16), (16, 16, 8), (31, 2, 17),
                                (32, 32, 32), (4, 32, 1)])
def test_sub_grid_sizes(ctx, built, n2):
    gpv = built
    tris = gpv.gen_torus(5, 40, 24, (0.5, 0.5, 0.5), 0.35, 0.12, 0.02)
    mn, mx = gpv.mesh_bounds(tris)
    _check(ctx, gpv, tris, gpv.grid_padded(mn, mx, (9, 10, 11), n2))


@pytest.mark.parametrize("shift,scale", [((0, 0, 0), 1.0), ((1000.0, -3000.0, 517.0), 1.0), ((3e5, 1e5, -2e5), 1.0),
                                         ((0, 0, 0), 3e-10), ((0, 0, 0), 2e10), ((-0.5, -0.5, -0.5), 1.0)])
def test_magnitudes(ctx, built, shift, scale):
    gpv = built
    tris = gpv.gen_uvsphere(9, 24, 12, (0.5, 0.5, 0.5), 0.4, 0.01).reshape(-1, 3)
    tris = np.ascontiguousarray(tris * np.float32(scale) + np.asarray(shift, np.float32), np.float32).reshape(-1)
    mn, mx = gpv.mesh_bounds(tris)
    _check(ctx, gpv, tris, gpv.grid_padded(mn, mx, 8, (6, 8, 5)))


@pytest.mark.parametrize("n1,n2", [((5, 6, 40), (16, 16, 16)), ((30, 30, 30), (8, 8, 8)), ((3, 3, 3), (32, 32, 32))])
def test_large_triangles(ctx, built, n1, n2):
    # a rotated box of 12 triangles and slivers through many voxels: every voxel of a column shares
    # its triangles, and rows run over whole voxels
    gpv = built
    rng = np.random.default_rng(3)
    c = np.array([[x, y, z] for x in (0, 1) for y in (0, 1) for z in (0, 1)], np.float64) - 0.5
    f = [(0, 1, 3), (0, 3, 2), (4, 6, 7), (4, 7, 5), (0, 4, 5), (0, 5, 1), (2, 3, 7), (2, 7, 6), (0, 2, 6), (0, 6, 4),
         (1, 5, 7), (1, 7, 3)]
    q, _ = np.linalg.qr(rng.normal(size=(3, 3)))
    box = (c @ q.T)[np.array(f)]
    sliver = rng.uniform(-0.4, 0.4, (6, 3, 3))
    sliver[:, 2] = sliver[:, 1] + rng.normal(size=(6, 3)) * 1e-4
    tris = np.ascontiguousarray(np.concatenate([box, sliver]), np.float32).reshape(-1)
    mn, mx = gpv.mesh_bounds(tris)
    _check(ctx, gpv, tris, gpv.grid_padded(mn, mx, n1, n2))


@pytest.mark.parametrize("n2", [(32, 32, 1), (32, 32, 32), (31, 32, 5), (16, 32, 8)])
def test_full_column_lists(ctx, built, n2):
    # near-horizontal sheets wider than the grid: each triangle leaves (nearly) all sub-columns of its
    # voxels, so one triangle fills the list of a batch and the others wait for the next
    gpv = built
    z = np.array([0.11, 0.12, 0.48, 0.48, 0.83])
    quad = np.array([[[-9, -9, 0], [9, -9, 0], [9, 9, 0]], [[-9, -9, 0], [9, 9, 0], [-9, 9, 0]]], np.float64)
    t = np.concatenate([quad + [0, 0, v] for v in z])
    t[4:] += t[4:, :, :1] * [0, 0, 0.013] + t[4:, :, 1:2] * [0, 0, 0.007]
    tris = np.ascontiguousarray(t, np.float32).reshape(-1)
    _check(ctx, gpv, tris, _spec(gpv, (0, 0, 0), (1, 1, 1), [2, 3, 4], list(n2)))
