"""The separate viscous kernel at every split of a block over a cluster (8, 4, 2
and 1 CTAs for 8, 120, 240 and 450 blocks), with UP ghosts (two-stage solver)
and with the zero ghosts of the single-stage solvers, against the oracle:
1e-10 relative L1 per conserved variable; the next step's dt likewise."""
import dataclasses

import numpy as np
import pytest

from walicxe3d_b200 import config as C
from walicxe3d_b200 import problems
from walicxe3d_b200.mesh import BlockTree, cell_centres

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("solver", [C.SOLVER_HLLC, C.SOLVER_HLL1])
@pytest.mark.parametrize("nroot", [(2, 2, 2), (4, 5, 6), (6, 5, 8), (9, 10, 5)])
def test_cluster_split_matches_oracle(nroot, solver):
    import oracle
    from walicxe3d_b200.solver import from_problem
    prob = problems.smooth_pulse(2, solver=solver)
    cfg = dataclasses.replace(prob.cfg, nbroot=nroot, box=tuple(n / 10.0 for n in nroot), visc_eta=0.02)
    tree = BlockTree(nroot, 1).roots()
    ids = np.asarray(tree.morton_order(), np.int32)
    x = cell_centres(cfg, tree, ids)
    p = np.zeros((len(ids), 5, 16, 16, 16))
    p[:, 0] = 1.0 + 0.3 * np.sin(9.0 * x[:, 0]) * np.cos(7.0 * x[:, 1] + 2.0 * x[:, 2])
    p[:, 1] = 0.2 * np.cos(8.0 * x[:, 2])
    p[:, 4] = 1.0 + 0.4 * np.cos(6.0 * x[:, 1]) * np.sin(5.0 * x[:, 2])
    prob = problems.Problem("split", cfg, tree, ids, problems.prim2flow(cfg, p))
    o = oracle.from_problem(prob, threads=8)
    g = from_problem(prob)
    g.set_fusion(False)
    for _ in range(4):
        o.step()
        g.step()
    ug, uo = g.download(), o.U[:len(ids)]
    assert g.state.dt == pytest.approx(o.state.dt, rel=1e-10)
    g.close()
    for e in range(5):
        assert np.abs(ug[:, e] - uo[:, e]).sum() <= 1e-10 * np.abs(uo[:, e]).sum(), e
