"""predictor_kernel and corrector_kernel at every launch shape (slabs of 16, 8,
4 and 2 planes, the viscous step fused and separate) and equation count,
on a three-level mesh (same, coarser, finer and boundary faces, both boundary
conditions) against the oracle: 1e-10 relative L1 per conserved variable."""
import dataclasses

import numpy as np
import pytest

from walicxe3d_b200 import config as C
from walicxe3d_b200 import problems

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("npassive", [0, 1, 2])
@pytest.mark.parametrize("solver,limiter,bc", [(C.SOLVER_HLLC, C.LIMITER_MINMOD, C.BC_FREE_FLOW),
                                               (C.SOLVER_HLL, C.LIMITER_UMIST, C.BC_REFLECTIVE),
                                               (C.SOLVER_HLLC, C.LIMITER_VANLEER, C.BC_FREE_FLOW),
                                               (C.SOLVER_HLL, C.LIMITER_WOODWARD, C.BC_REFLECTIVE)])
def test_every_launch_shape_matches_oracle(npassive, solver, limiter, bc):
    import oracle
    from walicxe3d_b200.solver import from_problem
    prob = problems.blast_amr(nroot=2, maxlev=3, shell_radius=0.1, shell_width=0.02, solver=solver, limiter=limiter)
    prob.cfg = dataclasses.replace(prob.cfg, npassive=npassive, bc=(bc,) * 6)
    rho = prob.U[:, :1]
    extra = [rho * (0.2 + 0.1 * k) * (1.0 + 0.3 * np.sin(7.0 * rho + k)) for k in range(npassive)]
    prob.U = np.ascontiguousarray(np.concatenate([prob.U] + extra, axis=1))
    o = oracle.from_problem(prob, threads=8)
    for _ in range(6):
        o.step()
    uo = o.U[:prob.nblocks]
    for zsplit, fused in ((1, True), (1, False), (2, False), (4, False), (8, False)):
        g = from_problem(prob)
        g.set_zsplit(zsplit)
        g.set_fusion(fused)
        for _ in range(6):
            g.step()
        ug = g.download()
        g.close()
        for e in range(prob.cfg.neqtot):
            assert np.abs(ug[:, e] - uo[:, e]).sum() <= 1e-10 * np.abs(uo[:, e]).sum(), (zsplit, fused, e)
