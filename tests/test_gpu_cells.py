"""Level1 cells of vertices where the estimate from the reciprocal must hand over to the quotient: a few
ulps around every cell boundary, at and just below the box's maximum (whose own cell steps down), outside
the box, and boxes of tiny, huge and uneven extents.  States, indices and the SAT count equal the
oracle's."""
import numpy as np
import pytest

from oracle import oracle as orc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lo,hi", [((0, 0, 0), (1, 1, 1)), ((-3.3, 0.1, 100), (7.7, 0.1001, 101)),
                                   ((1e-12, 0, -1e-12), (3e-12, 1e-12, 1e-12)), ((-1e18, -2e18, 0), (1e18, 2e18, 3e18)),
                                   ((1000, 1000, 1000), (1000.01, 1000.02, 1000.5))])
@pytest.mark.parametrize("n", [(1, 1, 1), (7, 10, 13), (64, 50, 33)])
def test_vertices_at_cell_boundaries(ctx, built, lo, hi, n):
    gpv = built
    rng = np.random.default_rng(sum(n))
    lo32, hi32 = np.asarray(lo, np.float32), np.asarray(hi, np.float32)
    m = 400
    v = np.empty((m, 3, 3), np.float32)
    for a in range(3):
        k = rng.integers(0, n[a] + 1, (m, 3))
        x = (lo32[a] + (hi32[a] - lo32[a]) * (k / n[a]).astype(np.float32)).astype(np.float32)
        for _ in range(3):
            x = np.where(rng.random(x.shape) < 0.5, np.nextafter(x, rng.choice([-np.inf, np.inf], x.shape).astype(np.float32)), x)
        x = np.where(rng.random(x.shape) < 0.1, hi32[a], x)
        x = np.where(rng.random(x.shape) < 0.05, lo32[a] - (hi32[a] - lo32[a]) * np.float32(0.3), x)
        # (small triangles: the corners of one share their neighbourhood)
        near = rng.random(m) < 0.7
        x[near, 1] = np.nextafter(x[near, 0], np.float32(np.inf))
        x[near, 2] = x[near, 0]
        v[:, :, a] = x
    tris = np.ascontiguousarray(v).reshape(-1)
    s = gpv.GridSpec()
    s.bbox_min[:] = [float(x) for x in lo32]
    s.bbox_max[:] = [float(x) for x in hi32]
    s.ndiv[:] = list(n)
    s.ndiv2[:] = [0, 0, 0]
    ref = orc.Run(tris, s, fill=orc.FILL_CAND)
    res = ctx.voxelize_host(tris, s)
    l1, pre, bi, _ = ctx.fetch(res)
    np.testing.assert_array_equal(l1, ref.level1_bytes())
    np.testing.assert_array_equal(pre, ref.prefix())
    np.testing.assert_array_equal(bi, ref.boundary_index())
    assert res.work.sat1 == ref.sat1_tests()
    ctx.release(res)
