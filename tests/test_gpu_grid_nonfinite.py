"""Walls and fixed cells of a file grid where a temperature is infinite or NaN,
in FAST mode: a wall's T reaches no other cell, and a fixed cell keeps its own
whatever its neighbours hold, as in the reference (eph_fdm.h:322-387).  Against
the oracle, finite cells at the bar of tests/test_gpu_grid_fast.py."""
import numpy as np
import pytest

import ephgb
from ephgb import workloads as W
from helpers import atom_err
from oracle.bindings import OracleFix

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [(8, 6, 5), (24, 23, 25)])  # in one cluster, in launches
@pytest.mark.parametrize("where", ["walls", "fixed", "inside"])
def test_nonfinite_cells(built, beta_file, tmp_path, n, where):
    at = W.fcc_lattice(5, seed=9)
    words = W.fix_args(beta_file, flags=4, grid=(1, 1, 1), T_infile=W.write_grid_file(str(tmp_path / "T.in"), n=n, seed=3))
    ref, fix = OracleFix(words, at, 0.001), ephgb.FixEPH(words, at, dt=0.001)
    nc = int(np.prod(n))
    i, j, k = np.arange(nc) % n[0], np.arange(nc) // n[0] % n[1], np.arange(nc) // (n[0] * n[1])
    T = np.random.default_rng(5).uniform(200.0, 3000.0, nc)
    wall, fixed = i == 0, (i > 0) & (j == 0) & (k == 0)
    if where == "walls":
        T[wall] = np.where(np.arange(wall.sum()) % 2, np.nan, np.inf)
    elif where == "fixed":
        T[fixed & (i == 2)] = np.inf
    else:
        T[(i == n[0] // 2) & (j == n[1] // 2) & (k == n[2] // 2)] = np.nan
    ref.set("T", T)
    fix.put("T", T)
    ref.step(np.zeros(3 * at.n))
    fix.step(1)
    got, want = fix.get("T"), ref.get("T")
    ok = np.isfinite(want)
    assert ok.any() and np.array_equal(np.isfinite(got), ok)
    assert np.array_equal(got[~ok & (wall | fixed)], want[~ok & (wall | fixed)], equal_nan=True)
    assert atom_err(got[ok], want[ok]) <= 1e-12
