"""wx3d_pack_blocks and wx3d_unpack_blocks: one block, around the slots one
launch takes (511, 512, 513), all blocks, an 8-byte aligned buffer, a slot
named twice (the last copy stays) and a slot out of range (nothing moves)."""
import ctypes

import numpy as np
import pytest

from walicxe3d_b200 import config as C

pytestmark = pytest.mark.gpu
IP = ctypes.POINTER(ctypes.c_int32)


@pytest.fixture(scope="module", params=[0, 1])
def loaded(request):
    from walicxe3d_b200.solver import Walicxe3D
    cfg = C.Config(npassive=request.param, nbroot=(10, 10, 6))
    w = Walicxe3D(cfg, 600)
    w.set_mesh(np.arange(1, 601, dtype=np.int32))
    u = np.random.default_rng(3).random((600, cfg.neqtot, 16, 16, 16)) + 1.0
    w.upload(u)
    yield w, u
    w.close()


def _call(w, f, slots, t):
    s = np.ascontiguousarray(slots, np.int32)
    return f(w.ctx, 0, len(s), s.ctypes.data_as(IP), ctypes.c_void_p(t.data_ptr()))


@pytest.mark.parametrize("n", [1, 511, 512, 513, 600])
@pytest.mark.parametrize("shift", [0, 1])
def test_round_trip(loaded, n, shift):
    import torch
    w, u = loaded
    w.upload(u)
    slots = np.random.default_rng(n).permutation(600)[:n]
    flat = torch.zeros(n * u[0].size + shift, dtype=torch.float64, device="cuda")
    buf = flat[shift:]
    assert _call(w, w.lib.wx3d_pack_blocks, slots, buf) == 0
    assert np.array_equal(buf.cpu().numpy(), u[slots].ravel())
    buf.mul_(2.0)
    torch.cuda.synchronize()
    assert _call(w, w.lib.wx3d_unpack_blocks, slots, buf) == 0
    expect = u.copy()
    expect[slots] *= 2.0
    assert np.array_equal(w.download(), expect)


def test_repeated_and_bad_slots(loaded):
    import torch
    w, u = loaded
    w.upload(u)
    buf = torch.rand((3, u[0].size), dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    assert _call(w, w.lib.wx3d_unpack_blocks, [7, 9, 7], buf) == 0
    got = w.download()
    assert np.array_equal(got[7].ravel(), buf[2].cpu().numpy()) and np.array_equal(got[9].ravel(), buf[1].cpu().numpy())
    assert _call(w, w.lib.wx3d_unpack_blocks, [3, 600], buf) == 103
    assert np.array_equal(w.download(), got)
    assert _call(w, w.lib.wx3d_pack_blocks, [5, 5], buf) == 0
    assert np.array_equal(buf[:2].cpu().numpy(), np.stack([got[5].ravel()] * 2))
