"""Level1 cells of triangles that leave an explicit box: a vertex just under the box's maximum whose
quotient rounds up to n, one exactly at the maximum (whose own cell steps down to n - 1) and one beyond
it, on each axis and in every vertex order, and random triangles that leave the box on every side.
States and indices equal the oracle's on the plain and the no-alloc path, and the SAT count the ranges
of the three vertices' cells (the oracle counts a triangle that misses the box by its empty range)."""
import ctypes as C
import itertools

import numpy as np
import pytest

from oracle import oracle as orc

pytestmark = pytest.mark.gpu

BOXES = [((-1, -1, -1), (1, 1, 1), (8, 8, 8)), ((-100, -100, -100), (0, 0, 0), (64, 64, 64)),
         ((-100, -1, -33), (0, 1, 0), (8, 50, 33)), ((-1e6, -1e-3, -1e3), (0, 0, 0), (16, 8, 4))]


def _spec(gpv, lo, hi, n):
    s = gpv.GridSpec()
    s.bbox_min[:] = [float(np.float32(v)) for v in lo]
    s.bbox_max[:] = [float(np.float32(v)) for v in hi]
    s.ndiv[:] = list(n)
    s.ndiv2[:] = [0, 0, 0]
    return s


def _sat1(tris, spec):
    v, f = tris.reshape(-1, 3, 3), np.float32
    count = np.ones(len(v), np.int64)
    for a in range(3):
        lo, hi, n = f(spec.bbox_min[a]), f(spec.bbox_max[a]), spec.ndiv[a]
        c = np.clip((v[:, :, a] - lo) / (hi - lo) * f(n), f(-1), f(n) + f(1)).astype(np.int64)
        c -= (c == n) & (v[:, :, a] == hi)
        count *= np.maximum(np.minimum(c.max(1), n - 1) - np.maximum(c.min(1), 0) + 1, 0)
    return int(count.sum())


def _check(ctx, gpv, tris, spec):
    import torch

    ref = orc.Run(tris, spec, fill=orc.FILL_CAND)
    res = ctx.voxelize_host(tris, spec)
    l1, pre, bi, _ = ctx.fetch(res)
    np.testing.assert_array_equal(l1, ref.level1_bytes())
    np.testing.assert_array_equal(pre, ref.prefix())
    np.testing.assert_array_equal(bi, ref.boundary_index())
    assert res.work.sat1 == _sat1(tris, spec)
    ctx.release(res)
    d = torch.from_numpy(tris).cuda()
    out = [torch.full((l1.size,), -1, dtype=t, device="cuda") for t in (torch.int8, torch.int32, torch.int32)]
    b = C.c_int64()
    rc = gpv.lib().gpv_voxelize_level1_noalloc(d.data_ptr(), tris.size // 9, C.byref(spec), out[0].data_ptr(),
                                               out[1].data_ptr(), out[2].data_ptr(), C.byref(b), 0)
    assert rc == 0, gpv.lib().gpv_noalloc_last_error()
    assert b.value == len(bi)
    np.testing.assert_array_equal(out[0].cpu().numpy().view(np.uint8), l1)
    np.testing.assert_array_equal(out[1].cpu().numpy(), pre)
    np.testing.assert_array_equal(out[2].cpu().numpy()[:b.value], bi)
    return ref.B


def _just_under(lo, hi, n):
    """The largest coordinates under hi whose quotient times n rounds to n."""
    lo, hi = np.float32(lo), np.float32(hi)
    out, x = [], np.nextafter(hi, lo)
    for _ in range(3):
        if np.float32((x - lo) / (hi - lo)) * np.float32(n) == n:
            out.append(x)
        x = np.float32(hi - 4 * max(hi - x, np.float32(np.spacing(np.float32(abs(hi - lo))) / 64)))
    return out


@pytest.mark.parametrize("box", range(len(BOXES)))
@pytest.mark.parametrize("axis", [0, 1, 2])
def test_under_at_and_beyond_the_maximum(ctx, built, box, axis):
    gpv = built
    lo, hi, n = BOXES[box]
    unders = _just_under(lo[axis], hi[axis], n[axis])
    assert unders
    tris = []
    for under in unders:
        beyond = np.float32(hi[axis] + 0.25 * (hi[axis] - lo[axis]))
        for order in itertools.permutations([under, np.float32(hi[axis]), beyond]):
            for u, v in ((0.3, 0.4), (0.6, 0.7)):
                t = np.empty((3, 3), np.float32)
                for a in range(3):
                    w = hi[a] - lo[a]
                    t[:, a] = [lo[a] + u * w, lo[a] + (u + 0.6 / n[a]) * w, lo[a] + v * w]
                t[:, axis] = order
                tris.append(t)
    tris = np.ascontiguousarray(tris, np.float32).reshape(-1)
    spec = _spec(gpv, lo, hi, n)
    # each triangle alone, so that none stands in for another, and all of them
    assert sum(_check(ctx, gpv, tris[9 * k:9 * k + 9].copy(), spec) for k in range(12)) > 0
    assert _check(ctx, gpv, tris, spec) > 0


@pytest.mark.parametrize("box", range(len(BOXES)))
@pytest.mark.parametrize("size", [0.02, 0.5])
def test_triangles_leave_the_box(ctx, built, box, size):
    gpv = built
    lo, hi, n = (np.asarray(v, np.float64) for v in BOXES[box])
    rng = np.random.default_rng([box, int(100 * size)])
    m = 600
    c = rng.uniform(-0.2, 1.2, (m, 1, 3))
    x = (lo + (hi - lo) * (c + rng.normal(size=(m, 3, 3)) * size)).astype(np.float32)
    # a fifth of the coordinates at, or a few ulps around, the faces
    lo32, hi32 = lo.astype(np.float32), hi.astype(np.float32)
    at = rng.random(x.shape)
    face = np.where(at < 0.1, lo32, hi32)
    step = rng.integers(-2, 3, x.shape).astype(np.float32) * np.spacing(np.abs(hi32 - lo32)) / 8
    x = np.where(at < 0.2, face + np.where(rng.random(x.shape) < 0.5, step, 0), x).astype(np.float32)
    spec = _spec(gpv, lo, hi, n.astype(int))
    assert _check(ctx, gpv, np.ascontiguousarray(x).reshape(-1), spec) > 0
