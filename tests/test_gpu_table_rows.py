"""The table lookup's guessed row: evenly spaced rows (the guess is the row or
next to it), rows crowded at either end (bisection takes over), and the
smallest tables, against the oracle's scan: 1e-10 relative L1 per variable."""
import numpy as np
import pytest

from walicxe3d_b200 import config as C
from walicxe3d_b200 import problems

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows", [2, 3, 50, 200])
@pytest.mark.parametrize("power", [1.0, 3.0, 0.3])
def test_any_row_spacing_matches_oracle(rows, power):
    import oracle
    from walicxe3d_b200.solver import from_problem
    prob = problems.cooling_blob(C.COOL_TABLE, nroot=2)
    logT = 4.0 + 3.2 * np.linspace(0.0, 1.0, rows) ** power   # the hottest cells lie above the last row
    prob.cooltable = (logT, 21.6 + 0.9 * (logT - 5.3) ** 2 / (1.0 + 0.35 * np.abs(logT - 5.3)))
    o = oracle.from_problem(prob, threads=8)
    g = from_problem(prob)
    for _ in range(4):
        o.step()
        g.step()
    ug, uo = g.download(), o.U[:prob.nblocks]
    g.close()
    for e in range(prob.cfg.neqtot):
        assert np.abs(ug[:, e] - uo[:, e]).sum() <= 1e-10 * np.abs(uo[:, e]).sum(), e
