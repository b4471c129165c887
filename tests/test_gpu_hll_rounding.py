"""One first-order HLL step of a state that varies along x, against the
reference's formulas in 80-bit arithmetic: the mean error of the mass and of
each momentum is no larger than that of the same formulas in IEEE 64-bit
arithmetic (both round each operation to half an ulp; 5 % for the sampling of
2,000 cells).  Slow flow is the hard case: the two sides' contributions cancel."""
import numpy as np
import pytest

from walicxe3d_b200 import config as C

pytestmark = pytest.mark.gpu
NB = 128   # blocks along x


def _flux(F, l, r, g, cv):
    """primfhll (hll.f90:175-260) of primitives [5, n]."""
    cl, cr = np.sqrt(g * l[4] / l[0]), np.sqrt(g * r[4] / r[0])
    sl, sr = np.minimum(l[1] - cl, r[1] - cr), np.maximum(l[1] + cl, r[1] + cr)

    def both(p):
        e = F(0.5) * p[0] * (p[1] * p[1] + p[2] * p[2] + p[3] * p[3]) + cv * p[4]
        u = np.stack([p[0], p[0] * p[1], p[0] * p[2], p[0] * p[3], e])
        return u, np.stack([p[0] * p[1], p[0] * p[1] * p[1] + p[4], p[0] * p[1] * p[2], p[0] * p[1] * p[3],
                            p[1] * (e + p[4])])
    (ul, fl), (ur, fr) = both(l), both(r)
    mid = (sr * fl - sl * fr + sl * sr * (ur - ul)) / (sr - sl)
    return np.where(sl >= 0, fl, np.where(sr <= 0, fr, mid))


def _step(F, u, dt, dx, g):
    """Conserved variables [5, n] of the interior cells after one step."""
    u, cv = u.astype(F), 1 / (F(g) - 1)
    rinv = 1 / u[0]   # the kernel's flow2prim: products by 1/rho and 1/cv
    v = u[1:4] * rinv
    p = (u[4] - F(0.5) * (u[1] * u[1] + u[2] * u[2] + u[3] * u[3]) * rinv) * (1 / cv)
    q = np.stack([u[0], v[0], v[1], v[2], p])
    f = _flux(F, q[:, :-1], q[:, 1:], F(g), cv)
    return u[:, 1:-1] + F(dt) / F(dx) * (f[:, :-1] - f[:, 1:])


@pytest.mark.parametrize("mach", [0.01, 0.3, 3.0])
def test_hll_step_rounds_like_ieee_arithmetic(mach):
    from walicxe3d_b200.solver import Walicxe3D
    cfg = C.Config(solver_type=C.SOLVER_HLL1, limiter_type=C.LIMITER_MINMOD, nbroot=(NB, 1, 1),
                   box=(1.0, 1.0 / NB, 1.0 / NB), visc_eta=0.0)
    rs = np.random.RandomState(4)
    n = NB * 16
    # a smooth walk, neighbours 0.1 % apart
    walk = lambda k: np.convolve(rs.uniform(-1, 1, n + 64), np.ones(64) / 8.0, "valid")[:n] * k   # noqa: E731
    rho, p = 1.0 + 0.1 * np.tanh(walk(0.1)), 1.0 + 0.1 * np.tanh(walk(0.1))
    c = np.sqrt(cfg.gamma)
    v = [mach * c * (0.6 + 0.2 * np.tanh(walk(0.2))) for _ in range(3)]
    cells = np.stack([rho, rho * v[0], rho * v[1], rho * v[2],
                      cfg.cv * p + 0.5 * rho * (v[0] ** 2 + v[1] ** 2 + v[2] ** 2)])
    u = np.ascontiguousarray(np.broadcast_to(cells.reshape(5, NB, 1, 1, 16).transpose(1, 0, 2, 3, 4), (NB, 5, 16, 16, 16)))
    w = Walicxe3D(cfg, NB)
    w.set_mesh(np.arange(1, NB + 1, dtype=np.int32))
    w.upload(u)
    w.set_state(it=20)
    dt = w.step().dt
    out = w.download()
    w.close()
    row = out[:, :, 8, 8, :].transpose(1, 0, 2).reshape(5, n)[:, 1:-1]
    assert np.array_equal(out, np.broadcast_to(out[:, :, 8:9, 8:9, :], out.shape))   # still a function of x
    dx = cfg.dx(1)[0]
    true = _step(np.longdouble, cells, dt, dx, cfg.gamma)
    ieee = _step(np.float64, cells, dt, dx, cfg.gamma)
    for e in range(4):
        assert np.abs(row[e] - true[e]).mean() <= 1.05 * np.abs(ieee[e] - true[e]).mean(), e
