"""A COOL_TABLE context finds a table laid out for its lookup whichever 180-row
loader filled it: the rows given as a Schure table or as a plain one cool alike
(the lookup's slopes lay past the end of the Schure table's memory)."""
import numpy as np
import pytest

from walicxe3d_b200 import config as C
from walicxe3d_b200 import problems

pytestmark = pytest.mark.gpu


def test_the_two_loaders_lay_out_the_same_table():
    from walicxe3d_b200.solver import from_problem
    prob = problems.cooling_blob(C.COOL_TABLE, nroot=2, steps=1)
    first = np.linspace(3.0, 9.0, 180)                       # the first column after the loader's power of ten
    second = 0.5 + 0.4 * np.cos(2.0 * first)                 # the second column, likewise: ten to it is the coefficient
    data = np.zeros((180, 5))
    data[:, 0], data[:, 1] = np.log10(first), -np.log10(second)
    out = []
    for plain in (True, False):
        w = from_problem(prob)
        if plain:
            w.set_cooltable(first, -second)
        else:
            w.set_cooltable_schure(data, 1)
        w.set_state(it=20, dt=1.5e-28)
        w.sources()
        out.append(w.download())
        w.close()
    change = 1.0 - out[0][:, 4] / prob.U[:, 4]
    assert 1e-3 < change.max() < 0.45   # cooled, and not clipped
    np.testing.assert_allclose(out[1], out[0], rtol=1e-12)
