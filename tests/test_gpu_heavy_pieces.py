"""Pieces of large triangles: their places in the list are taken for a warp's triangles together.  Warps that
mix small and large triangles, triangles that go to several meshes of a batch, and more pieces than the
list holds (a triangle that fits partly stays with its group).  States equal the oracle's."""
import numpy as np
import pytest

from oracle import oracle as orc

pytestmark = pytest.mark.gpu


def _soup(n, size, seed):
    rng = np.random.default_rng(seed)
    c = rng.uniform(0, 1, (n, 1, 3))
    s = np.broadcast_to(np.asarray(size), (n,)).reshape(-1, 1, 1)
    return np.ascontiguousarray((c + rng.normal(size=(n, 3, 3)) * s).astype(np.float32)).reshape(-1)


def _spec(gpv, n):
    s = gpv.GridSpec()
    s.bbox_min[:], s.bbox_max[:], s.ndiv[:], s.ndiv2[:] = [0.0] * 3, [1.0] * 3, list(n), [0] * 3
    return s


def _equal(ctx, res, tris, spec):
    ref = orc.Run(tris, spec, fill=orc.FILL_CAND)
    l1, pre, bi, _ = ctx.fetch(res)
    np.testing.assert_array_equal(l1, ref.level1_bytes())
    np.testing.assert_array_equal(pre, ref.prefix())
    np.testing.assert_array_equal(bi, ref.boundary_index())
    assert res.num_pairs == int(ref.L.orc_num_pairs(ref.h))


@pytest.mark.parametrize("n", [1, 31, 33, 700])
def test_small_and_large_in_a_warp(ctx, built, n):
    import torch

    gpv = built
    rng = np.random.default_rng(n)
    meshes = [(_soup(k, np.where(rng.random(k) < 0.4, 0.3, 0.005), k), _spec(gpv, g))
              for k, g in ((n, (70, 64, 50)), (2 * n + 5, (33, 90, 40)), (n + 1, (128, 9, 64)))]
    dev = [torch.from_numpy(t).cuda() for t, _ in meshes]
    torch.cuda.synchronize()
    res = ctx.voxelize_batch([d.data_ptr() for d in dev], [d.numel() // 9 for d in dev], [s for _, s in meshes])
    for r, (t, s) in zip(res, meshes):
        _equal(ctx, r, t, s)
        ctx.release(r)


def test_more_pieces_than_the_list_holds(ctx, built):
    gpv = built
    tris, spec = _soup(80000, 0.25, 5), _spec(gpv, (72, 64, 8))
    v = tris.reshape(-1, 3, 3)
    span = [np.clip(np.floor(v[:, :, a].max(1) * spec.ndiv[a]), 0, spec.ndiv[a] - 1)
            - np.clip(np.floor(v[:, :, a].min(1) * spec.ndiv[a]), 0, spec.ndiv[a] - 1) + 1 for a in range(2)]
    assert (span[0] * span[1] // 128).sum() > 1 << 18  # (the SAT units alone)
    res = ctx.voxelize_host(tris, spec)
    _equal(ctx, res, tris, spec)
    ctx.release(res)
