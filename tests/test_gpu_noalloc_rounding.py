"""eph_fdm_solve_noalloc rounds like the reference's source expressions
(EPH_FDM::solve, eph_fdm.h:315-396): every bit of T against a numpy restatement
in their order.  Grids with walls, fixed cells and sources, axes of one cell
and odd sizes; spacings, conductivities and temperatures over many binades;
zeros, from which every quotient is zero, and tiny values, whose products leave
the range of the integer arithmetic."""
import ctypes as C

import numpy as np
import pytest

import ephgb
from test_zz_no_alloc import _device_grid, _solve

pytestmark = pytest.mark.gpu


def solve(g, n, lo, hi, dt, nsub):
    """nsub substeps of EPH_FDM::solve, one rounding per operation"""
    shape = (n[2], n[1], n[0])
    T, kappa, flag = g["T"].reshape(shape), g["kappa"].reshape(shape), g["flag"].reshape(shape)
    S, dT = g["S"].reshape(shape), g["dT"].reshape(shape)
    rhoC = g["rho"].reshape(shape) * g["C"].reshape(shape)
    inner = dt / nsub
    for _ in range(nsub):
        dd = np.zeros(shape)
        for axis, h in ((2, (hi[0] - lo[0]) / n[0]), (1, (hi[1] - lo[1]) / n[1]), (0, (hi[2] - lo[2]) / n[2])):
            wq, wp = np.roll(flag, -1, axis) == 2, np.roll(flag, 1, axis) == 2
            wp &= ~wq
            Tq, kq = np.where(wq, T, np.roll(T, -1, axis)), np.where(wq, kappa, np.roll(kappa, -1, axis))
            Tp, kp = np.where(wp, T, np.roll(T, 1, axis)), np.where(wp, kappa, np.roll(kappa, 1, axis))
            dd = dd + (kq - kp) * (Tq - Tp) / h / h / 4.0
            dd = dd + kappa * ((Tq + Tp - 2.0 * T) / h / h)
        new = T + (dd + dT + S) / rhoC * inner
        T = np.where(flag == 1, new, T)
        T = np.where(T < 0.0, 0.0, T)
    return T.ravel()


CASES = [((12, 10, 8), "plain", 0.002), ((1, 1, 1), "plain", 0.001), ((33, 1, 5), "walls", 0.001), ((17, 19, 23), "walls", 0.002),
         ((64, 64, 64), "walls", 0.002), ((16, 9, 11), "zeros", 0.001), ((16, 9, 11), "tiny", 0.001)]


@pytest.mark.parametrize("n,what,dt", CASES)
def test_every_bit(built, n, what, dt):
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(7)
    nt = n[0] * n[1] * n[2]
    g = dict(T=rng.uniform(1.0, 3000.0, nt), S=rng.uniform(-50.0, 50.0, nt) * (rng.random(nt) < 0.2), dT=rng.uniform(-5.0, 5.0, nt),
             rho=rng.uniform(0.5, 1.5, nt), C=rng.uniform(1e-6, 5e-6, nt), kappa=rng.uniform(0.01, 0.2, nt),
             flag=np.ones(nt, dtype=np.int8))
    if what == "walls":
        i, j = np.arange(nt) % n[0], np.arange(nt) // n[0] % n[1]
        g["flag"][i == 0] = 2
        g["flag"][(j == 0) & (i > 0)] = 0
        g["flag"][rng.random(nt) < 0.05] = 2
    if what == "zeros":
        g["T"][rng.random(nt) < 0.5] = 0.0
        g["kappa"][rng.random(nt) < 0.5] = 0.0
        g["S"][:] = g["dT"][:] = 0.0
    if what == "tiny":
        g["T"] *= 10.0 ** rng.uniform(-300.0, 3.0, nt)
        g["kappa"] *= 10.0 ** rng.uniform(-150.0, 0.0, nt)
        g["S"][:] = 0.0
        g["dT"] *= 10.0 ** rng.uniform(-300.0, 0.0, nt)
    lo, hi = np.array([0.0, -5.0, 1.0]), np.array([0.0, -5.0, 1.0]) + np.array([3.4, 3.7, 3.1]) * n
    d = _device_grid(g, torch)
    d["dT"] = torch.tensor(g["dT"], dtype=torch.float64, device="cuda:0")
    nsub = C.c_uint()
    assert _solve(d, n, lo, hi, dt, 1, nsub) == ephgb.EPH_OK
    want = solve(g, n, lo, hi, dt, nsub.value)
    got = d["T"].cpu().numpy()
    assert np.array_equal(got, want), (int((got != want).sum()), float(np.abs(got - want).max()))
