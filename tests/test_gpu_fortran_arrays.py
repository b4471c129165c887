"""The Fortran-array transfers with fewer, as many and more array entries than
block slots, from pageable and pinned memory: every physical cell of the
entries that exist travels, every ghost and every other entry stays."""
import numpy as np
import pytest

from walicxe3d_b200 import config as C

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nbmax", [1, 7, 16, 20, 33])
@pytest.mark.parametrize("pinned", [False, True])
def test_only_physical_cells_travel(nbmax, pinned):
    import torch
    from walicxe3d_b200.solver import Walicxe3D
    w = Walicxe3D(C.Config(npassive=1, nbroot=(2, 2, 2)), 20)
    w.set_mesh(np.arange(1, 9, dtype=np.int32))
    ns = min(nbmax, 20)

    def array(values):
        t = torch.from_numpy(np.ascontiguousarray(values))   # [k][j][i][eq][nb]
        return (t.pin_memory() if pinned else t).numpy()
    start = np.random.default_rng(5).random((20, 6, 16, 16, 16))
    w.upload(start)
    up = array(np.random.default_rng(6).random((20, 20, 20, 6, nbmax)))
    w.upload_fortran(up.T)
    native = w.download(20)
    expect = start.copy()
    expect[:ns] = up[2:18, 2:18, 2:18, :, :ns].transpose(4, 3, 0, 1, 2)
    assert np.array_equal(native, expect)
    down = array(np.full((20, 20, 20, 6, nbmax), -7.0))
    w.download_fortran(down.T)
    want = np.full_like(down, -7.0)
    want[2:18, 2:18, 2:18, :, :ns] = up[2:18, 2:18, 2:18, :, :ns]
    assert np.array_equal(down, want)
    w.close()
