"""A few large triangles on tall grids: walls, whose units run through all layers and come in pieces of one
chunk of units where their boxes have more than 32 layers, and faces and slopes in pieces of four.  Every
output equals the oracle's, on the plain call and on the no-alloc entry."""
import ctypes as C

import numpy as np
import pytest

from oracle import oracle as orc

pytestmark = pytest.mark.gpu


def _box(tilt):
    v = np.array([[x, y, z] for x in (0, 1) for y in (0, 1) for z in (0, 1)], np.float64) * 0.7 + 0.15
    v[:, 0] += tilt * v[:, 2]
    f = [(0, 1, 3), (0, 3, 2), (4, 6, 7), (4, 7, 5), (0, 4, 5), (0, 5, 1), (2, 3, 7), (2, 7, 6), (0, 2, 6),
         (0, 6, 4), (1, 5, 7), (1, 7, 3)]
    return v[np.array(f)].astype(np.float32).reshape(-1)


@pytest.mark.parametrize("tilt", [0.0, 0.3])
@pytest.mark.parametrize("n", [(40, 36, 31), (40, 36, 47), (40, 36, 48), (90, 70, 200), (300, 4, 64)])
def test_outputs(ctx, built, tilt, n):
    gpv = built
    torch = pytest.importorskip("torch")

    tris = _box(tilt)
    spec = gpv.grid_padded(*gpv.mesh_bounds(tris), n, 2)
    ref = orc.Run(tris, spec, fill=orc.FILL_CAND)
    res = ctx.voxelize_host(tris, spec)
    l1, pre, bi, l2 = ctx.fetch(res)
    assert res.num_pairs == ref.num_pairs()
    ctx.release(res)
    np.testing.assert_array_equal(l1, ref.level1_bytes())
    np.testing.assert_array_equal(pre, ref.prefix())
    np.testing.assert_array_equal(bi, ref.boundary_index())
    np.testing.assert_array_equal(l2, ref.level2_bytes())

    dev, n1 = torch.from_numpy(tris).cuda(), n[0] * n[1] * n[2]
    a = torch.zeros(n1, dtype=torch.uint8, device="cuda")
    p = torch.zeros(n1, dtype=torch.int32, device="cuda")
    x = torch.zeros(n1, dtype=torch.int32, device="cuda")
    b = C.c_int64()
    rc = gpv.lib().gpv_voxelize_level1_noalloc(dev.data_ptr(), tris.size // 9, C.byref(spec), a.data_ptr(),
                                               p.data_ptr(), x.data_ptr(), C.byref(b),
                                               torch.cuda.current_stream().cuda_stream)
    assert rc == 0 and b.value == ref.B
    np.testing.assert_array_equal(a.cpu().numpy(), ref.level1_bytes())
    np.testing.assert_array_equal(p.cpu().numpy(), ref.prefix())
    np.testing.assert_array_equal(x.cpu().numpy()[:ref.B], ref.boundary_index())
