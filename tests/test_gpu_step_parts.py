"""wx3d_step_part after steps made another way: the stages of a part take every
block again, however the steps before it were launched (one call per step, a
replayed graph, or a part that was begun and left)."""
import ctypes

import numpy as np
import pytest

from walicxe3d_b200 import config as C
from walicxe3d_b200 import problems

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("solver", [C.SOLVER_HLLC, C.SOLVER_HLL1])
@pytest.mark.parametrize("steps", [2, 3])
def test_parts_after_a_replayed_graph_equal_parts_after_single_steps(solver, steps):
    from walicxe3d_b200.solver import from_problem
    prob = problems.smooth_pulse(nroot=8, solver=solver)   # 512 blocks: more items than one wave of CTAs
    states = []
    for replay in (True, False):
        w = from_problem(prob)
        w.set_zsplit(1)
        part = lambda k: w._chk(w.lib.wx3d_step_part(w.ctx, k), "wx3d_step_part")  # noqa: E731
        w.run(2)
        dtmin = ctypes.c_double()
        w._chk(w.lib.wx3d_get_dtmin(w.ctx, ctypes.byref(dtmin)), "wx3d_get_dtmin")
        part(0)   # begun, and left
        w._chk(w.lib.wx3d_set_dtmin(w.ctx, dtmin), "wx3d_set_dtmin")
        if replay:
            w.run(steps)
        else:
            for _ in range(steps):
                w.step()
        for k in (1, 2, 3):
            part(k)
        states.append(w.download())
        w.close()
    assert np.array_equal(states[0], states[1])
