"""The no-alloc entry reports a bounded wait that gave up instead of returning incomplete states, and the
calls after it are whole again."""
import ctypes as C

import numpy as np
import pytest

from oracle import oracle as orc

pytestmark = pytest.mark.gpu

WAIT_LIMIT, FAIL_WAIT, ERR_DEVICE = 1, 2, -6


def test_wait_gives_up(built):
    import torch

    gpv = built
    tris = gpv.gen_uvsphere(11, 64, 32, (0.5, 0.5, 0.5), 0.4, 0.002)
    spec = gpv.grid_padded(*gpv.mesh_bounds(tris), (40, 33, 37))
    ref = orc.Run(tris, spec, fill=orc.FILL_CAND)
    d = torch.from_numpy(tris).cuda()
    n1 = 40 * 33 * 37
    l1 = torch.zeros(n1, dtype=torch.uint8, device="cuda")
    pre, idx = (torch.zeros(n1, dtype=torch.int32, device="cuda") for _ in range(2))
    L, b = gpv.lib(), C.c_int64(-1)

    def call():
        return L.gpv_voxelize_level1_noalloc(d.data_ptr(), tris.size // 9, C.byref(spec), l1.data_ptr(),
                                             pre.data_ptr(), idx.data_ptr(), C.byref(b), 0)

    def whole():
        assert call() == 0, L.gpv_noalloc_last_error()
        assert b.value == ref.B
        np.testing.assert_array_equal(l1.cpu().numpy(), ref.level1_bytes())
        np.testing.assert_array_equal(pre.cpu().numpy(), ref.prefix())
        np.testing.assert_array_equal(idx.cpu().numpy()[:ref.B], ref.boundary_index())

    whole()
    assert L.gpv_noalloc_set_debug(FAIL_WAIT, 1) == 0
    try:
        b.value = -1
        assert call() == ERR_DEVICE
        assert b"wait" in L.gpv_noalloc_last_error() and b.value == -1
    finally:
        L.gpv_noalloc_set_debug(FAIL_WAIT, 0)
    whole()
    L.gpv_noalloc_set_debug(WAIT_LIMIT, 1 << 20)
    try:
        whole()
    finally:
        L.gpv_noalloc_set_debug(WAIT_LIMIT, 0)
    assert L.gpv_noalloc_set_debug(99, 1) != 0 and L.gpv_noalloc_set_debug(FAIL_WAIT, -1) != 0
