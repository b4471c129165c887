"""Every wave region of the branch-free HLLC and HLL fluxes against the oracle:
supersonic to either side, subsonic with the contact moving either way, two
colliding and two receding streams, at rest, and sound speeds far below the
flow speed.  Bar: 1e-10 relative L1 per conserved variable, as in the other
parity tests; a state at rest stays exactly at rest."""
import numpy as np
import pytest

from walicxe3d_b200 import config as C
from walicxe3d_b200 import problems

pytestmark = pytest.mark.gpu

REGIONS = {  # (rho, u, p) left, right
    "supersonic+": ((1.0, 6.0, 1.0), (0.5, 5.0, 0.4)),
    "supersonic-": ((0.5, -5.0, 0.4), (1.0, -6.0, 1.0)),
    "contact+": ((1.0, 0.2, 1.0), (0.125, 0.0, 0.1)),
    "contact-": ((0.125, 0.0, 0.1), (1.0, -0.2, 1.0)),
    "colliding": ((1.0, 3.0, 0.5), (0.7, -3.0, 0.6)),
    "receding": ((1.0, -1.0, 0.4), (1.0, 1.0, 0.4)),
    "cold": ((1.0, 8.0, 1.0e-4), (2.0, 7.0, 1.0e-4)),
    "rest": ((1.0, 0.0, 1.0), (1.0, 0.0, 1.0)),
}


@pytest.mark.parametrize("solver", [C.SOLVER_HLLC, C.SOLVER_HLL])
@pytest.mark.parametrize("region", sorted(REGIONS))
def test_flux_region_matches_oracle(region, solver):
    import oracle
    from walicxe3d_b200.solver import from_problem
    left, right = REGIONS[region]
    prob = problems.shock_tube(nblocks=2, axis=sorted(REGIONS).index(region) % 3, left=left, right=right, solver=solver)
    o = oracle.from_problem(prob, threads=2)
    g = from_problem(prob)
    for _ in range(12):
        o.step()
        g.step()
    ug, uo = g.download(), o.U[:prob.nblocks]
    g.close()
    if region == "rest":
        assert np.array_equal(ug, prob.U)
    for e in range(prob.cfg.neqtot):
        ref = np.abs(uo[:, e]).sum()
        diff = np.abs(ug[:, e] - uo[:, e]).sum()
        assert diff <= 1e-10 * ref if ref > 0 else diff == 0.0
