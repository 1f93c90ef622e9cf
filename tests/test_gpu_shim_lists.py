"""CUDAClassifyTessellationLevel2's sums where the order of a list matters: lists longer than a batch,
triangles that share sub-columns in one batch, sub-grids of one cell, of long rows and of more than 32
layers, empty lists, and arrays that already hold values.  Each cell's sum equals a float sum in list
order over the triangles that pass the reference's test."""
import ctypes as C

import numpy as np
import pytest

from oracle import oracle as orc
from test_gpu_shims import F3, I3, _setup

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n2", [(4, 4, 4), (1, 1, 1), (2, 3, 40), (33, 5, 3)])
def test_sums_in_list_order(built, n2):
    torch = pytest.importorskip("torch")
    L = built.lib()
    _setup(built, L)
    rng = np.random.default_rng(sum(n2))
    lens = [70, 0, 5, 33]
    B, cells = len(lens), int(np.prod(n2))
    f32 = np.float32
    e1 = np.array([0.5, 0.5, 0.5], f32)
    e2 = (e1 / np.array(n2, f32)).astype(f32)
    mid = rng.uniform(-1, 1, (B, 3)).astype(f32)
    tris = []
    for b, n in enumerate(lens):
        c = mid[b] + rng.uniform(-0.55, 0.55, (n, 1, 3))
        tris.append(c + rng.normal(size=(n, 3, 3)) * rng.choice([0.02, 0.3], (n, 1, 1)))
    tris = np.concatenate(tris).astype(f32).reshape(-1, 9)
    start = np.concatenate([[0], np.cumsum(lens)[:-1]]).astype(np.int32)
    flat = rng.permutation(len(tris)).astype(np.int32)  # (any triangles, in any order)
    l2 = np.where(rng.random(B * cells) < 0.5, 1.0, 0.0).astype(f32)
    nrm = rng.normal(size=(B * cells, 4)).astype(f32)
    want_l2, want = l2.copy(), nrm.copy()
    for b in range(B):
        cen = [[f32((p + 0.5) * float(f32(e2[a] * f32(2))) + float(mid[b, a]) - float(e1[a])) for p in range(n2[a])]
               for a in range(3)]
        for t in flat[start[b]:start[b] + lens[b]]:
            tv, fn = tris[t], orc.face_normal(tris[t])
            lo, hi = tv.reshape(3, 3).min(0), tv.reshape(3, 3).max(0)
            ok = [[i for i in range(n2[a]) if cen[a][i] + 1.5 * e2[a] >= lo[a] and cen[a][i] - 1.5 * e2[a] <= hi[a]]
                  for a in range(3)]
            for r in ok[2]:
                for q in ok[1]:
                    for p in ok[0]:
                        if orc.tri_box(np.array([cen[0][p], cen[1][q], cen[2][r]], f32), e2, tv):
                            o = b * cells + (r * n2[1] + q) * n2[0] + p
                            want_l2[o] = 2
                            want[o, :3] += np.asarray(fn, f32)
                            want[o, 3] += f32(1)
    d = [torch.from_numpy(x).cuda() for x in (tris.reshape(-1), l2, nrm.reshape(-1), mid.reshape(-1),
                                              np.arange(B, dtype=np.int32), np.array(lens, np.int32), start, flat)]
    rc = L.CUDAClassifyTessellationLevel2(*[x.data_ptr() for x in d], B, I3(*n2), F3(*[float(v) for v in e1]),
                                          F3(*[float(v) for v in e2]))
    assert rc == 1
    np.testing.assert_array_equal(d[1].cpu().numpy(), want_l2)
    np.testing.assert_array_equal(d[2].cpu().numpy().reshape(-1, 4), want)
