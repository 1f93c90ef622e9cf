"""Level2 work items where their starts and ends can go wrong: columns longer than a chunk and than a
mask word, column bits that start inside a word, chunks cut by z slabs, and batches with meshes that
have no boundary voxels or no Level2 grid (sorted for their normals, or not at all) between others.
States are decisions, so every byte equals the oracle's."""
import numpy as np
import pytest

from oracle import oracle as orc

pytestmark = pytest.mark.gpu


def _spec(gpv, n, n2):
    s = gpv.GridSpec()
    s.bbox_min[:] = [-0.1, -0.1, -0.1]
    s.bbox_max[:] = [1.4, 1.2, 1.1]
    s.ndiv[:] = list(n)
    s.ndiv2[:] = list(n2)
    return s


def _walls(seed):
    # upright and slanted sheets and a few small triangles: full columns, gaps, single voxels
    rng = np.random.default_rng(seed)
    a = rng.uniform(0.1, 0.9, (5, 2))
    t = [[[x, y, 0.02], [x + 0.3, y + 0.1, 0.03], [x + 0.15, y + 0.05, 0.97]] for x, y in a]
    s = rng.uniform(0.1, 0.9, (40, 1, 3)) + rng.normal(size=(40, 3, 3)) * 0.01
    return np.ascontiguousarray(np.concatenate([np.array(t), s]), np.float32).reshape(-1)


@pytest.mark.parametrize("nz", [1, 31, 32, 33, 77])
@pytest.mark.parametrize("chunk,slabs", [(32, 0), (1, 0), (5, 3), (32, 8)])
@pytest.mark.parametrize("fill", ["ray", "stencil"])
def test_columns_chunks_and_slabs(ctx, built, nz, chunk, slabs, fill):
    import torch

    gpv = built
    tris = _walls(nz)
    spec = _spec(gpv, (9, 7, nz), (3, 4, 5))
    n1, cells = 9 * 7 * nz, 60
    ref = orc.Run(tris, spec, fill=orc.FILL_CAND if fill == "ray" else orc.FILL_STENCIL)
    want = ref.level2_bytes()
    pin = [torch.empty(n, dtype=torch.uint8).pin_memory() for n in (n1, 4 * n1, 4 * n1, max(want.size, 1))]
    h = torch.from_numpy(tris).pin_memory()
    ctx.set_fill(gpv.FILL_RAY if fill == "ray" else gpv.FILL_STENCIL)
    ctx.set_level2_chunk(chunk)
    try:
        rc, res = ctx.voxelize_to_host(h.data_ptr(), tris.size // 9, spec, *[p.data_ptr() for p in pin], want.size,
                                       slabs)
        assert rc == 0 and res.num_boundary * cells == want.size
        np.testing.assert_array_equal(pin[3].numpy()[:want.size], want)
        np.testing.assert_array_equal(ctx.fetch(res)[3], want)
        ctx.release(res)
    finally:
        ctx.set_level2_chunk(32)
        ctx.set_fill(gpv.FILL_RAY)


@pytest.mark.parametrize("normals", [False, True])
def test_batch_of_unlike_meshes(ctx, built, normals):
    import torch

    gpv = built
    far = np.full(18, 50, np.float32)  # outside its grid: no boundary voxels
    cases = [(far, (4, 4, 4), (2, 2, 2)), (_walls(1), (9, 7, 33), (3, 4, 5)), (far, (4, 4, 4), (2, 2, 2)),
             (_walls(2), (11, 5, 40), (0, 0, 0)), (_walls(3), (3, 3, 3), (8, 8, 8)), (_walls(4), (16, 16, 70), (2, 3, 2)),
             (far, (5, 4, 4), (0, 0, 0))]
    specs = [_spec(gpv, a, b) for _, a, b in cases]
    dev = [torch.from_numpy(t).cuda() for t, _, _ in cases]
    ctx.set_normals(gpv.NORMALS_FLOAT if normals else gpv.NORMALS_OFF)
    try:
        for _ in range(2):
            rs = ctx.voxelize_batch([d.data_ptr() for d in dev], [d.numel() // 9 for d in dev], specs)
            for (t, _, b), s, r in zip(cases, specs, rs):
                ref = orc.Run(t, s, fill=orc.FILL_CAND)
                l1, _, bi, l2 = ctx.fetch(r)
                np.testing.assert_array_equal(l1, ref.level1_bytes())
                np.testing.assert_array_equal(bi, ref.boundary_index())
                if b[0]:
                    np.testing.assert_array_equal(l2, ref.level2_bytes())
                ctx.release(r)
    finally:
        ctx.set_normals(gpv.NORMALS_OFF)


@pytest.mark.parametrize("n2", [(4, 4, 8), (8, 4, 8), (4, 12, 8), (8, 8, 8), (16, 16, 8), (32, 32, 8), (4, 4, 16),
                                (8, 8, 16), (12, 8, 16), (16, 32, 16)])
@pytest.mark.parametrize("where", ["device", "direct", "packed"])
def test_output_units(ctx, built, n2, where):
    # one unit of 16 sub-columns a voxel to 64, powers of two and not, in device memory, written to the
    # host as bytes, and as packed codes for the first half of every slab's voxels
    import torch

    gpv = built
    tris = _walls(9)
    spec = _spec(gpv, (9, 7, 11), n2)
    want = orc.Run(tris, spec, fill=orc.FILL_CAND).level2_bytes()
    if where == "device":
        res = ctx.voxelize_host(tris, spec)
        np.testing.assert_array_equal(ctx.fetch(res)[3], want)
        ctx.release(res)
        return
    n1 = 9 * 7 * 11
    pin = [torch.empty(n, dtype=torch.uint8).pin_memory() for n in (n1, 4 * n1, 4 * n1, want.size)]
    h = torch.from_numpy(tris).pin_memory()
    if where == "packed":
        ctx.set_host_expand(2, 0xff, 50, 0)
    try:
        for _ in range(2):
            pin[3].fill_(77)
            rc, res = ctx.voxelize_to_host(h.data_ptr(), tris.size // 9, spec, *[p.data_ptr() for p in pin], want.size, 0)
            assert rc == 0
            np.testing.assert_array_equal(pin[3].numpy(), want)
            ctx.release(res)
    finally:
        ctx.set_host_expand()
