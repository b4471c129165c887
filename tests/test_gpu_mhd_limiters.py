"""MHD correctors with a limiter other than minmod -- van Leer, compiled in, and
Superbee and UMIST by the run-time switch -- fused with the viscous step and in
slabs, against the oracle: 1e-10 relative L1 of the density, the energy and the
two vectors.  A component is measured against its vector: rounding in the
fluxes goes with the vector's size, and the tube's B_z and m_z vanish but for
2e-6 that the viscous step brings in through the block-face ghosts."""
import numpy as np
import pytest

from walicxe3d_b200 import config as C
from walicxe3d_b200 import problems

pytestmark = pytest.mark.gpu


def _tube():
    return problems.brio_wu(8)


def _refined_vortex():
    return problems.orszag_tang_3d(nroot=4, flux_cd=False, maxlev=2)


@pytest.mark.parametrize("make", [_tube, _refined_vortex])
@pytest.mark.parametrize("solver", [C.SOLVER_HLLD, C.SOLVER_HLLE, C.SOLVER_HLL])
@pytest.mark.parametrize("limiter", [C.LIMITER_VANLEER, C.LIMITER_SUPERBEE, C.LIMITER_UMIST])
def test_mhd_limiter_matches_oracle(make, solver, limiter):
    import oracle
    from walicxe3d_b200.solver import from_problem
    prob = make()
    prob.cfg.solver_type = solver
    prob.cfg.limiter_type = limiter
    prob.cfg.visc_eta = 5.0e-3
    o = oracle.from_problem(prob, threads=8)
    for _ in range(12):
        o.step()
    uo = o.U[:prob.nblocks]
    for zsplit, fused in ((1, True), (1, False), (4, False)):
        g = from_problem(prob)
        g.set_zsplit(zsplit)
        g.set_fusion(fused)
        for _ in range(12):
            g.step()
        ug = g.download()
        g.close()
        for e in range(prob.cfg.neqtot):
            size = uo[:, 1:4] if 1 <= e <= 3 else (uo[:, 5:8] if e >= 5 else uo[:, e])
            assert np.abs(ug[:, e] - uo[:, e]).sum() <= 1e-10 * np.abs(size).sum(), (zsplit, fused, e)
