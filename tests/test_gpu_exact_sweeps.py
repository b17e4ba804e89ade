"""EXACT mode bit for bit against the oracle on its first step, at the sizes
where its lanes per atom change, with atoms in any order (the candidate sort),
more candidates than the shared-memory rows hold, operands that the integer
products and quotients leave to the hardware (zeros, tiny and huge values), and
its grid solve on both sides of the cluster's size."""
import numpy as np
import pytest

import ephgb
from ephgb import workloads as W
from helpers import n_in_group, xi_rows
from oracle.bindings import OracleFix

pytestmark = pytest.mark.gpu
KEYS = ("rho", "w", "f_eph", "f_rng", "f", "x", "v", "array")


def check(words, at, scale_xi=1.0, deposit=True):
    """deposit False: the forces alone, of the hooks before end_of_step (the
    energies of huge velocities are outside the deposits' fixed-point range,
    and refused)"""
    gpu, ref = ephgb.FixEPH(words, at, dt=0.001, mode=ephgb.MODE_EXACT), OracleFix(words, at, 0.001)
    stream = scale_xi * W.gaussian_stream(n_in_group(at), 9, 0)
    if deposit:
        gpu.step(1, xi=xi_rows(at, stream))
    else:
        gpu.initial_integrate()
        gpu.put("f", np.zeros((at.n, 3)))
        gpu.post_force(xi=xi_rows(at, stream))
        gpu.final_integrate()
    ref.step(stream)
    for k in KEYS:
        assert np.array_equal(gpu.get(k), ref.get(k)), k


def shuffle(at, seed):
    order = np.random.default_rng(seed).permutation(at.n)
    for name in ("x", "v", "type", "mask"):
        setattr(at, name, np.ascontiguousarray(getattr(at, name)[order]))
    return at


# cells (4 atoms each; 16^3 is the first size with fewer lanes), lattice
# constant, elements, flags
CASES = [((5, 5, 5), 3.52, 1, 7), ((6, 5, 7), 3.52, 2, 7), ((6, 6, 6), 2.75, 1, 7), ((6, 6, 6), 2.75, 2, 7),
         ((16, 15, 17), 3.52, 2, 7), ((16, 16, 16), 3.52, 1, 7), ((17, 16, 16), 3.52, 2, 5), ((20, 21, 10), 2.75, 1, 7)]


@pytest.mark.parametrize("shuffled", [False, True])
@pytest.mark.parametrize("cells,a,elements,flags", CASES)
def test_first_step_bitwise(built, beta_file, beta_file_2el, cells, a, elements, flags, shuffled):
    at = W.fcc_lattice(cells, a=a, seed=71)
    rng = np.random.default_rng(5)
    if elements == 2:
        at.type = np.where(rng.random(at.n) < 0.4, 2, 1).astype(np.int32)
        at.mass = np.array([0.0, W.NI_MASS, 55.845])
        at.mask = np.where(rng.random(at.n) < 0.1, 2, 1).astype(np.int32)
    if shuffled:
        at = shuffle(at, 3)
    words = W.fix_args(beta_file_2el if elements == 2 else beta_file, flags=flags, grid=(5, 4, 6), T_e=700.0,
                       elements=("Ni", "Fe")[:elements])
    check(words, at)


@pytest.mark.parametrize("v_scale,xi_scale", [(0.0, 1.0), (1e-300, 1e-290), (1e170, 1e160), (1.0, 0.0)])
def test_values_left_to_the_hardware(built, beta_file, v_scale, xi_scale):
    at = W.fcc_lattice((5, 5, 6), jitter=0.0, seed=7)  # the lattice's own zeros in x_j - x_i
    at.v = at.v * v_scale
    # NVE off (0x08): velocities of this size would leave the box
    check(W.fix_args(beta_file, flags=7 | 0x08 | 0x10 | 0x20, grid=(3, 3, 3), T_e=700.0), at, xi_scale, deposit=False)


# one cell per thread: a partial warp, a full cluster (16 x 512 cells), one past it
@pytest.mark.parametrize("grid", [(1, 1, 2), (3, 5, 7), (9, 7, 13), (16, 32, 16), (16, 32, 17)])
@pytest.mark.parametrize("walls", [False, True])
def test_grid_solve_bitwise(built, beta_file, tmp_path, grid, walls):
    atoms = W.fcc_lattice(5, seed=9)
    words = W.fix_args(beta_file, flags=4, grid=grid)
    if walls:
        if min(grid) < 3:
            pytest.skip("walls need three cells per axis")
        words = W.fix_args(beta_file, flags=4, grid=(1, 1, 1),
                           T_infile=W.write_grid_file(str(tmp_path / "T.in"), n=grid, seed=3))
    ref, fix = OracleFix(words, atoms, 0.001), ephgb.FixEPH(words, atoms, dt=0.001, mode=ephgb.MODE_EXACT)
    T = np.random.default_rng(5).uniform(0.0, 3000.0, int(np.prod(grid)))
    T[::7] = 300.0
    ref.set("T", T)
    fix.put("T", T)
    for _ in range(2):
        ref.step(np.zeros(3 * atoms.n))
        fix.step(1)
    assert np.array_equal(fix.get("T"), ref.get("T"))
