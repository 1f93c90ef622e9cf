"""Boxes so small that the inverse of their extent or of a Level2 cell overflows: cells and their ranges then
come from the quotient and from the exact tests.  Triangles inside the box, on its low faces, and large
ones that cross it.  Extents and divisions are powers of two, so that halving a cell is exact among the
denormals too and the oracle's centre tables are the library's.  Every state equals the oracle's."""
import numpy as np
import pytest

from oracle import oracle as orc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("span", [2.0 ** -124, 2.0 ** -121, 2.0 ** -118, 2.0 ** -110])
@pytest.mark.parametrize("n2", [(0, 0, 0), (1, 1, 1), (4, 4, 4), (8, 2, 8)])
@pytest.mark.parametrize("low", [0.0, -0.5])
def test_states(ctx, built, span, n2, low):
    gpv = built
    rng = np.random.default_rng(int(-np.log10(span)))
    m, n = 400, (64, 8, 16)
    v = rng.uniform(0, 1, (m, 1, 3)) + rng.normal(size=(m, 3, 3)) * 0.05
    v[rng.random((m, 3, 3)) < 0.15] = 0.0                    # low faces
    v[:40] = rng.uniform(-1, 2, (40, 3, 3))                  # large against the box
    v = (v + low) * span
    v[40:60] = rng.uniform(-1, 1, (20, 3, 3))                # ... and against everything
    v[40:60, :, 2] *= span
    tris = np.ascontiguousarray(v.astype(np.float32)).reshape(-1)
    spec = gpv.GridSpec()
    spec.bbox_min[:], spec.bbox_max[:] = [float(np.float32(low * span))] * 3, [float(np.float32((1 + low) * span))] * 3
    spec.ndiv[:], spec.ndiv2[:] = list(n), list(n2)
    ref = orc.Run(tris, spec, fill=orc.FILL_CAND)
    assert ref.B > 100
    for normals in (False, True):
        ctx.set_normals(gpv.NORMALS_FLOAT if normals else gpv.NORMALS_OFF)
        try:
            res = ctx.voxelize_host(tris, spec)
            l1, pre, bi, l2 = ctx.fetch(res)
            np.testing.assert_array_equal(l1, ref.level1_bytes())
            np.testing.assert_array_equal(pre, ref.prefix())
            np.testing.assert_array_equal(bi, ref.boundary_index())
            if n2[0]:
                np.testing.assert_array_equal(l2, ref.level2_bytes())
            if normals and n2[0]:
                np.testing.assert_array_equal(ctx.fetch_normals(res)[1], ref.level2_normals())
            ctx.release(res)
        finally:
            ctx.set_normals(gpv.NORMALS_OFF)
