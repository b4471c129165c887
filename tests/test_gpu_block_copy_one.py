"""Copying one block costs no more than the plain copy call that an 8-byte
aligned buffer takes (1.13 times as long when it took the kernel)."""
import ctypes
import time

import numpy as np
import pytest

from walicxe3d_b200 import config as C

pytestmark = pytest.mark.gpu


def test_one_block_is_a_plain_copy():
    import torch
    from walicxe3d_b200.solver import Walicxe3D
    w = Walicxe3D(C.Config(nbroot=(2, 2, 2)), 8)
    w.set_mesh(np.arange(1, 9, dtype=np.int32))
    u = np.random.default_rng(1).random((8, 5, 16, 16, 16)) + 1.0
    w.upload(u)
    flat = torch.zeros(u[0].size + 1, dtype=torch.float64, device="cuda")
    slot = np.array([3], np.int32)
    s = slot.ctypes.data_as(ctypes.POINTER(ctypes.c_int32))

    def took(shift):
        p = ctypes.c_void_p(flat[shift:].data_ptr())
        t = time.perf_counter()
        assert w.lib.wx3d_pack_blocks(w.ctx, 0, 1, s, p) == 0
        return time.perf_counter() - t
    times = {0: [], 1: []}
    for k in range(2000):
        times[k & 1].append(took(k & 1))
    assert np.array_equal(flat[1:].cpu().numpy(), u[3].ravel())
    w.close()
    assert np.median(times[0][100:]) <= 1.06 * np.median(times[1][100:])
