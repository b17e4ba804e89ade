"""The FAST grid substeps (precomputed coefficients; one cluster launch for
small grids, per-substep launches for larger ones) against the oracle.

Tolerance: a substep adds d to T; both sides round the sum once (2^-53 of T)
and d itself, whose terms are at most 0.8 T in all, in about ten operations, so
a substep differs by at most ~1e-15 T and the steps here (up to ~700 substeps)
by less than 1e-12 T, the bar of the other parity tests."""
import numpy as np
import pytest

import ephgb
from ephgb import workloads as W
from helpers import atom_err
from oracle.bindings import OracleFix

pytestmark = pytest.mark.gpu
TOL = 1e-12


def start_T(n, seed=5):
    return np.random.default_rng(seed).uniform(200.0, 3000.0, n)


# cells: fewer than a warp, axes of 1 and 2, a partial last block, the largest
# cluster grid (16 x 384 cells) and one past it, odd sizes on the launches
GRIDS = [(1, 1, 1), (2, 1, 3), (3, 5, 7), (9, 7, 13), (16, 24, 16), (16, 24, 17), (24, 23, 25)]


@pytest.mark.parametrize("grid", GRIDS)
@pytest.mark.parametrize("walls", [False, True])
def test_fast_solve_matches_the_oracle(built, beta_file, tmp_path, grid, walls):
    atoms = W.fcc_lattice(5, seed=9)
    words = W.fix_args(beta_file, flags=4, grid=grid)
    if walls:
        if min(grid) < 3:
            pytest.skip("walls need three cells per axis")
        words = W.fix_args(beta_file, flags=4, grid=(1, 1, 1),
                           T_infile=W.write_grid_file(str(tmp_path / "T.in"), n=grid, seed=3))
    ref, fix = OracleFix(words, atoms, 0.001), ephgb.FixEPH(words, atoms, dt=0.001)
    T = start_T(int(np.prod(grid)))
    ref.set("T", T)
    fix.put("T", T)
    xi = np.zeros(3 * atoms.n)
    for _ in range(2):
        ref.step(xi)
        fix.step(1)
    assert atom_err(fix.get("T"), ref.get("T")) <= TOL


@pytest.mark.parametrize("how", ["graph", "batch"])
def test_new_grid_constants_reach_captured_steps(built, beta_file, how):
    """set_grid_constants and reset_dt between captured steps give what a
    context built with those values gives (the coefficients follow, and so
    does the count of substeps)."""
    atoms = W.fcc_lattice(5, seed=9)

    def words(C, kappa):
        return W.fix_args(beta_file, flags=4, grid=(8, 7, 6), C_e=C, kappa_e=kappa)

    T = start_T(336)
    if how == "graph":
        fix = ephgb.FixEPH(words(3.5e-6, 0.1), atoms, dt=0.001)
        fix.set_graph(True)
        step, sync = fix.step, fix.synchronize
    else:
        batch = ephgb.Batch([(words(3.5e-6, 0.1), atoms)] * 2, dt=0.001)
        fix, step, sync = batch.replicas[1], batch.step, batch.synchronize
    step(2)
    sync()
    for C, kappa, dt in ((3.5e-6, 0.02, 0.001), (2e-6, 0.4, 0.001), (2e-6, 0.4, 0.0005)):
        fix.set_grid_constants(C, kappa)
        fix.reset_dt(dt)
        new = ephgb.FixEPH(words(C, kappa), atoms, dt=dt)
        for f in (fix, new):
            f.put("T", T)
            f.synchronize()
        step(3)
        sync()
        new.step(3)
        assert np.array_equal(fix.get("T"), new.get("T"))
