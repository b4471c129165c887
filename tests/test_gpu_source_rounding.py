"""One plain source step (hydrogen ionisation and cooling_h, or table cooling)
of cells over the whole range of temperatures, against the reference's formulas
in 80-bit arithmetic: the kernel's mean error is no larger than that of the same
formulas in IEEE 64-bit arithmetic.  Both round each operation to half an ulp,
so the means agree to the sampling error of 32,768 cells, under 1 % (5 % are
allowed); products by reciprocals or differences of logarithms in their place
leave a tenth to a third more."""
import numpy as np
import pytest

from walicxe3d_b200 import config as C

pytestmark = pytest.mark.gpu
PC, YR = C.PC, C.YR
RANGES = [(3.0, 4.0), (4.0, 4.6), (4.6, 5.0), (5.0, 6.0), (6.0, 8.0)]


def _cfg(cooling):
    return C.Config(npassive=1, eos_type=C.EOS_H_RATE, cooling_type=cooling, limiter_type=C.LIMITER_MINMOD,
                    nbroot=(2, 2, 2), box=(PC,) * 3, l_sc=PC, d_sc=1.3 * C.AMU, v_sc=1.0e5, tfin=1e30, dtout=1e30)


def _cells(cfg, lo, hi, seed):
    rs = np.random.RandomState(seed)
    shape = (8, 16, 16, 16)
    n, T, y = 10.0 ** rs.uniform(-1.5, 1.5, shape), 10.0 ** rs.uniform(lo, hi, shape), rs.uniform(1e-3, 0.999, shape)
    u = np.zeros((8, 6, 16, 16, 16))
    u[:, 0], u[:, 5] = n * cfg.mu0, n * y
    u[:, 4] = cfg.cv * n * (2.0 - y) * C.KB * T / cfg.p_sc   # at rest
    return u


def _ion(F, cfg, rho, p, nhi, s):
    """Neutral fraction after s seconds (hrate.f90:96-137)."""
    n = rho / F(cfg.mu0)
    T = p / (2 * n - nhi) * F(cfg.p_sc) / F(C.KB)
    xi, y0 = F(1e-4), nhi / n
    col = F(5.83e-11) * np.sqrt(T) * np.exp(F(-157828.0) / T)
    rec = F(2.55e-13) * np.exp(F(0.79) * np.log(F(1e4) / T))
    a, b, c = rec + col, -((2 + xi) * rec + (1 + xi) * col), (1 + xi) * rec
    d = np.sqrt(b * b - 4 * a * c)
    g = (2 * a * y0 + b + d) / (2 * a * y0 + b - d) * np.exp(-d * n * s)
    return np.maximum(np.minimum((-b - d * (1 + g) / (1 - g)) / (2 * a), 1 - xi), F(0))


def _loss(F, x1, den, h0, T):
    """cooling_h.f90:42-145 above 1e4 K."""
    hp = (1 - x1) * den
    de = hp + F(1e-4) * den
    lo = F(0.5732) + T * (F(1.8288e-5) + T * (F(-1.15822e-10) + T * F(9.4288e-16)))
    hi = F(0.5856) + T * (F(1.55083e-5) + T * (F(-9.669e-12) + T * F(5.716e-19)))
    w = (T - 55000) / F(17000)
    om = np.where(T <= 55000, lo, np.where(T >= 72000, hi, (1 - w) * lo + w * hi))
    s = np.sqrt(T)
    coll = np.maximum(de * h0 * (F(8.6287e-6) / (2 * s) * om * np.exp(F(-118409.0) / T)) * F(1.634e-11), F(0))
    ion = de * h0 * (F(5.834e-11) * s * np.exp(F(-1.579e5) / T)) * F(2.179e-11)
    q = F(157890.0) / T
    lq = np.log(q)
    rec = np.maximum(de * hp * (F(1.133e-24) / np.sqrt(q) * (F(-0.0713) + F(0.5) * lq + F(0.640) * np.exp(F(-0.33333) * lq))), F(0))
    t = 1 / T
    oi = de * (F(1e-3) * h0) * F(10) ** (F(1381465) * (t * t) - F(12328.69) * t - F(19.82621))
    oii = de * (F(1e-3) * hp) * F(10) ** (F(-2061075.0) * (t * t) - F(14596.24) * t - F(19.01402))
    eq = F(1.0455e-18) / np.exp(F(0.63) * np.log(T)) * (1 - np.exp(-np.exp(F(1.63) * np.log(T * F(1e-5))))) * de * den \
        + de * hp * (F(1.3) * F(1.42e-27) * s)
    x = np.exp(-2 * (np.clip(T, 44770, 54770) - 49770) / F(500))
    fr = np.where(T <= 44770, F(0), np.where(T >= 54770, F(1), F(0.5) * (1 + (1 - x) / (1 + x))))
    return coll + ion + (rec + F(7.033) * (oi + oii)) * (1 - fr) + eq * fr


def _step(F, cfg, table, u, s, nhi=None):
    """Neutral density and energy after the step, and where the energy changed freely; nhi given: the
    energy for that neutral density."""
    rho, e, h = (u[:, k].astype(F) for k in (0, 4, 5))
    p, s = e / F(cfg.cv), F(s)
    n = rho / F(cfg.mu0)
    new = n * _ion(F, cfg, rho, p, h, s) if nhi is None else nhi.astype(F)
    T = p / (2 * n - new) * F(cfg.p_sc) / F(C.KB)
    if table is None:
        hot = np.maximum(T, F(10001))
        L = _loss(F, F(cfg.mu0) * h / rho, n, new, hot)
        f = (10 + (hot - 10) * np.exp(-(2 * L / (3 * F(C.KB) * n * hot)) * s)) / hot
        free = T > 10001
    else:
        lt, c = table[0].astype(F), -table[1].astype(F)
        x = np.clip(np.log10(T), lt[0], lt[-1])
        i = np.clip(np.searchsorted(lt, x, side="right") - 1, 0, len(lt) - 2)
        lam = F(10) ** ((c[i + 1] - c[i]) / (lt[i + 1] - lt[i]) * (x - lt[i]) + c[i])
        nd = rho * F(cfg.d_sc) / (F(cfg.mui) * F(C.AMU))
        f = np.exp(-(lam * (nd * nd) / (F(cfg.cv) * p * F(cfg.p_sc))) * s)
        free = (np.log10(T) > lt[0]) & (np.log10(T) < lt[-1])
    return new, F(cfg.cv) * (p * f), free & (f > 0.51) & (f < 1)   # by way of the pressure, as the reference


def _table():
    lt = np.linspace(4.0, 9.0, 200)
    return lt, 21.6 + 0.9 * (lt - 5.3) ** 2 / (1.0 + 0.35 * np.abs(lt - 5.3)) - 0.25 * np.tanh(lt - 7.5)


@pytest.mark.parametrize("cooling", [C.COOL_H, C.COOL_TABLE])
@pytest.mark.parametrize("lo,hi", RANGES)
def test_source_step_rounds_like_ieee_arithmetic(cooling, lo, hi):
    from walicxe3d_b200.solver import Walicxe3D
    cfg = _cfg(cooling)
    table = _table() if cooling == C.COOL_TABLE else None
    u = _cells(cfg, lo, hi, 11)
    dt = 50.0 * YR / cfg.t_sc
    w = Walicxe3D(cfg, 8)
    w.set_mesh(np.arange(1, 9, dtype=np.int32))
    if table is not None:
        w.set_cooltable(*table)
    w.upload(u)
    w.set_state(it=20, dt=dt)
    w.sources()
    out = w.download()
    w.close()
    s, L = dt * cfg.t_sc, np.longdouble
    true_n = _step(L, cfg, table, u, s)[0]
    ieee_n = _step(np.float64, cfg, table, u, s)[0]
    n = u[:, 0] / cfg.mu0
    err = lambda a: float((np.abs(a - true_n) / n).mean())   # noqa: E731
    assert err(out[:, 5]) <= 1.05 * err(ieee_n)
    # the energy at the neutral density each side found
    errs = []
    for h, e in ((out[:, 5], out[:, 4]), (ieee_n, _step(np.float64, cfg, table, u, s, ieee_n)[1])):
        _, true_e, free = _step(L, cfg, table, u, s, h)
        if free.sum() < 2000:   # too few cells cool there (below 1e4 K)
            return
        errs.append(float((np.abs(e - true_e) / true_e)[free].mean()))
    assert errs[0] <= 1.05 * errs[1]
