"""Level1 outputs (states, boundaryPrefixSum, boundaryIndex) at row lengths where the expansion's words,
pieces and chunks end: rows shorter than a plane word, of one voxel, of a multiple of four or not, a word
and a piece more, and grids of part of a chunk to several.  Bytes and indices equal the oracle's."""
import numpy as np
import pytest

from oracle import oracle as orc

pytestmark = pytest.mark.gpu


def _case(gpv, n):
    s = gpv.GridSpec()
    s.bbox_min[:] = [0.0, 0.0, 0.0]
    s.bbox_max[:] = [1.0, 1.0, 1.0]
    s.ndiv[:] = list(n)
    s.ndiv2[:] = [0, 0, 0]
    return gpv.gen_torus(3, 40, 24, (0.5, 0.5, 0.5), 0.33, 0.13, 0.02), s


def _check(ctx, res, tris, spec):
    ref = orc.Run(tris, spec, fill=orc.FILL_CAND)
    l1, pre, bi, _ = ctx.fetch(res)
    np.testing.assert_array_equal(l1, ref.level1_bytes())
    np.testing.assert_array_equal(pre, ref.prefix())
    np.testing.assert_array_equal(bi, ref.boundary_index())
    assert res.num_level1_inside == int((l1 == 127).sum())


@pytest.mark.parametrize("nx", [1, 2, 3, 4, 5, 7, 8, 12, 28, 31, 32, 33, 36, 60, 64, 65, 100, 128])
@pytest.mark.parametrize("ny,nz", [(1, 1), (9, 13), (50, 41)])
def test_row_lengths(ctx, built, nx, ny, nz):
    tris, spec = _case(built, (nx, ny, nz))
    res = ctx.voxelize_host(tris, spec)
    _check(ctx, res, tris, spec)
    ctx.release(res)


def test_batch_of_row_lengths(ctx, built):
    import torch

    cases = [_case(built, n) for n in [(5, 9, 13), (32, 3, 3), (1, 1, 1), (64, 20, 20), (33, 7, 50), (4, 100, 3)]]
    dev = [torch.from_numpy(t).cuda() for t, _ in cases]
    rs = ctx.voxelize_batch([d.data_ptr() for d in dev], [d.numel() // 9 for d in dev], [s for _, s in cases])
    for (t, s), r in zip(cases, rs):
        _check(ctx, r, t, s)
        ctx.release(r)
