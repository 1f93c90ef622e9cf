"""The Level2 stencil fill's samples where their batches and edge functions can go wrong: one sub-cell to
32 per axis, triangles without samples between others, triangles far larger than a voxel (edge functions
beyond 32 bits, coordinates past the snapping clamp), vertices on sample centres, and columns longer than
a chunk.  States are decisions, so every byte equals the oracle's."""
import numpy as np
import pytest

from oracle import oracle as orc

pytestmark = pytest.mark.gpu


def _soup(kind):
    rng = np.random.default_rng(7)
    small = rng.uniform(0.1, 0.9, (300, 1, 3)) + rng.normal(size=(300, 3, 3)) * 0.03
    if kind == "small":
        return small
    if kind == "snapped":  # vertices on sample centres and cell corners of a 1/64 lattice
        return np.round(small * 64) / 64
    big = rng.normal(size=(8, 3, 3)) * np.array([3.0, 3.0, 0.4]) + 0.5
    if kind == "large":
        return np.concatenate([small[:50], big])
    return np.concatenate([small[:50], big * np.array([4e6, 4e6, 1.0])])  # "huge"


@pytest.mark.parametrize("n1,n2", [((5, 6, 40), (8, 8, 8)), ((4, 4, 4), (1, 1, 1)), ((3, 2, 9), (32, 32, 4)),
                                   ((4, 3, 5), (31, 7, 32)), ((2, 2, 70), (3, 5, 2))])
@pytest.mark.parametrize("kind", ["small", "snapped", "large", "huge"])
def test_samples(ctx, built, n1, n2, kind):
    gpv = built
    tris = np.ascontiguousarray(_soup(kind), np.float32).reshape(-1)
    s = gpv.GridSpec()
    s.bbox_min[:] = [0.0, 0.0, 0.0]
    s.bbox_max[:] = [1.0, 1.0, 1.0]
    s.ndiv[:] = list(n1)
    s.ndiv2[:] = list(n2)
    ctx.set_fill(gpv.FILL_STENCIL)
    try:
        res = ctx.voxelize_host(tris, s)
    finally:
        ctx.set_fill(gpv.FILL_RAY)
    ref = orc.Run(tris, s, fill=orc.FILL_STENCIL)
    l1, _, bi, l2 = ctx.fetch(res)
    np.testing.assert_array_equal(l1, ref.level1_bytes())
    np.testing.assert_array_equal(bi, ref.boundary_index())
    np.testing.assert_array_equal(l2, ref.level2_bytes())
    ctx.release(res)
