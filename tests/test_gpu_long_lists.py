"""Voxel lists put in triangle order: one long list among short ones, around the lengths where the sort
changes (a warp, a block's network, the block's bit map), several long lists, ids spread over more than
one pass of the bit map, and meshes of a batch.  Sums run in list order, so every normal equals the
oracle's."""
import numpy as np
import pytest

from oracle import oracle as orc

pytestmark = pytest.mark.gpu


def _cluster(n, at, seed):
    rng = np.random.default_rng(seed)
    c = rng.uniform(at, at + 1e-3, (n, 1, 3))
    return (c + rng.normal(size=(n, 3, 3)) * 1e-4).astype(np.float32)


def _mesh(gpv, lengths, seed, base=90):
    """A torus and clusters of tiny triangles, each inside one voxel, in random order."""
    t = [gpv.gen_torus(seed, 2 * base, base, (0.5, 0.5, 0.5), 0.35, 0.12, 0.004).reshape(-1, 3, 3)]
    t += [_cluster(n, 0.102 + 0.06 * k, seed + k) for k, n in enumerate(lengths)]
    t = np.concatenate(t)
    return np.ascontiguousarray(t[np.random.default_rng(seed).permutation(len(t))]).reshape(-1)


def _spec(gpv, n, n2):
    s = gpv.GridSpec()
    s.bbox_min[:], s.bbox_max[:], s.ndiv[:], s.ndiv2[:] = [-0.1] * 3, [1.1] * 3, [n] * 3, [n2] * 3
    return s


def _equal(ctx, res, tris, spec, longest):
    ref = orc.Run(tris, spec, fill=orc.FILL_CAND)
    _, _, bi, _ = ctx.fetch(res)
    np.testing.assert_array_equal(bi, ref.boundary_index())
    # the rule that picks this sort: at most 64 triangles a voxel on the average
    assert int(ref.L.orc_num_pairs(ref.h)) <= 64 * ref.B
    n1, n2 = ctx.fetch_normals(res)
    np.testing.assert_array_equal(n1, ref.level1_normals())
    if spec.ndiv2[0]:
        np.testing.assert_array_equal(n2, ref.level2_normals())
    assert longest is None or res.num_pairs > longest


@pytest.mark.parametrize("lengths", [(512,), (513,), (8192,), (8193,), (9000, 700, 20000, 8192), (33, 64, 65, 30000)])
@pytest.mark.parametrize("n2", [0, 2])
def test_list_lengths(ctx, built, lengths, n2):
    gpv = built
    tris, spec = _mesh(gpv, lengths, 3), _spec(gpv, 60, n2)
    ctx.set_normals(gpv.NORMALS_FLOAT)
    try:
        res = ctx.voxelize_host(tris, spec)
        _equal(ctx, res, tris, spec, max(lengths))
        ctx.release(res)
    finally:
        ctx.set_normals(gpv.NORMALS_OFF)


@pytest.mark.parametrize("extra", [0, 1])
def test_ids_of_several_passes(ctx, built, extra):
    gpv = built
    # 12 * 1024 * 32 ids a pass: the third pass holds one id, or 777
    base = gpv.gen_torus(4, 660, 330, (0.5, 0.5, 0.5), 0.35, 0.12, 0.004).size // 9
    n = 12 * 1024 * 32 + 1 - base if extra else 2 * 12 * 1024 * 32 + 777 - base
    if n <= 8192:
        n += 12 * 1024 * 32
    tris, spec = _mesh(gpv, (n,), 4, 330), _spec(gpv, 128, 0)
    ctx.set_normals(gpv.NORMALS_FLOAT)
    try:
        res = ctx.voxelize_host(tris, spec)
        _equal(ctx, res, tris, spec, n)
        ctx.release(res)
    finally:
        ctx.set_normals(gpv.NORMALS_OFF)


def test_batch(ctx, built):
    import torch

    gpv = built
    meshes = [(_mesh(gpv, ls, 10 + k), _spec(gpv, 60, n2))
              for k, (ls, n2) in enumerate((((9000,), 2), ((), 0), ((20000, 600), 2), ((8500,), 0)))]
    dev = [torch.from_numpy(t).cuda() for t, _ in meshes]
    torch.cuda.synchronize()
    ctx.set_normals(gpv.NORMALS_FLOAT)
    try:
        res = ctx.voxelize_batch([d.data_ptr() for d in dev], [d.numel() // 9 for d in dev], [s for _, s in meshes])
        for r, (t, s) in zip(res, meshes):
            _equal(ctx, r, t, s, None)
            ctx.release(r)
    finally:
        ctx.set_normals(gpv.NORMALS_OFF)
