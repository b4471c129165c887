"""Fortran-array transfers where the array has more entries than the context
has slots, or a few entries only: every way a plane can travel (whole rows, one
contiguous span, strided lines) gives the same cells and leaves the rest alone,
and none costs a multiple of what an array without the extra entries costs
(15 times when every such array took strided rows)."""
import time

import numpy as np
import pytest

from walicxe3d_b200 import config as C

pytestmark = pytest.mark.gpu
# slots, entries: single entry, small spans, misaligned and line-aligned strides, either side of 64 KB a plane
SIZES = [(1, 1), (1, 2), (2, 3), (3, 4), (3, 5), (4, 4), (5, 5), (5, 29), (8, 16), (16, 24), (12, 13), (33, 34)]


def _array(values, pinned, shift):
    import torch
    flat = torch.zeros(values.size + 16, dtype=torch.float64)
    flat = flat.pin_memory() if pinned else flat
    a = flat.numpy()[shift:shift + values.size].reshape(values.shape)   # [k][j][i][eq][nb]
    a[...] = values
    return a


@pytest.mark.parametrize("slots,nbmax", SIZES)
@pytest.mark.parametrize("pinned,shift", [(False, 0), (False, 2), (True, 0), (True, 1)])
def test_physical_cells_travel_and_nothing_else(slots, nbmax, pinned, shift):
    from walicxe3d_b200.solver import Walicxe3D
    w = Walicxe3D(C.Config(nbroot=(4, 3, 3)), slots)
    w.set_mesh(np.arange(1, slots + 1, dtype=np.int32) if slots == 36 else np.full(slots, -1, np.int32))
    rs = np.random.default_rng(slots * 100 + nbmax)
    w.upload(rs.random((slots, 5, 16, 16, 16)))
    up = _array(rs.random((20, 20, 20, 5, nbmax)), pinned, shift)
    w.upload_fortran(up.T)
    assert np.array_equal(w.download(slots), up[2:18, 2:18, 2:18, :, :slots].transpose(4, 3, 0, 1, 2))
    down = _array(np.full(up.shape, -7.0), pinned, shift)
    w.download_fortran(down.T)
    want = np.full_like(down, -7.0)
    want[2:18, 2:18, 2:18, :, :slots] = up[2:18, 2:18, 2:18, :, :slots]
    assert np.array_equal(down, want)
    w.close()


@pytest.mark.parametrize("slots,nbmax", [(3, 4), (5, 9), (7, 12), (33, 36), (65, 66)])
@pytest.mark.parametrize("pinned", [False, True])
def test_extra_entries_cost_no_multiple(slots, nbmax, pinned):
    from walicxe3d_b200.solver import Walicxe3D
    a = _array(np.random.default_rng(1).random((20, 20, 20, 5, nbmax)), pinned, 0)
    took = {}
    for n in (nbmax, slots):
        w = Walicxe3D(C.Config(nbroot=(5, 5, 5)), n)
        for name, call in (("up", w.upload_fortran), ("down", w.download_fortran)):
            t = []
            for _ in range(15):
                s = time.perf_counter()
                call(a.T)
                t.append(time.perf_counter() - s)
            took[n, name] = np.median(t)
        w.close()
    for name in ("up", "down"):
        assert took[slots, name] < 2.5 * took[nbmax, name] + 100e-6, (name, took)
