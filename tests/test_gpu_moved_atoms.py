"""Atoms that moved since the candidate lists were built, in the df64 sweeps:
fast atoms at the corners, edges and middle of the box, across the periodic
boundary and, over the steps, past many neighbours, against the oracle (1e-12
per atom, the parity tests' bar), with one lane and several per atom, and with
more moved atoms than are handled between two builds."""
import numpy as np
import pytest

import ephgb
from ephgb import workloads as W
from helpers import key_err, n_in_group, xi_rows
from oracle.bindings import OracleFix

pytestmark = pytest.mark.gpu
TOL = 1e-12
KEYS = ("rho", "w", "f_eph", "f_rng", "x", "v")


def hot_atoms(at, count, speed, seed):
    """`count` atoms, the corners' and faces' first, at `speed` A/ps"""
    rng = np.random.default_rng(seed)
    span = at.boxhi - at.boxlo
    spots = [np.array([i, j, k]) / 2.0 for i in (0, 1, 2) for j in (0, 1, 2) for k in (0, 1, 2)][:count]
    spots += [rng.random(3) for _ in range(count - len(spots))]
    for s in spots:
        d = at.x - (at.boxlo + s * span * (1 - 1e-9))
        i = int(np.argmin((d * d).sum(axis=1)))
        u = rng.standard_normal(3)
        at.v[i] = speed * u / np.sqrt((u * u).sum())


# cells, elements, lanes per atom (0: the rule), hot atoms, their speed
CASES = [((17, 16, 16), 1, 0, 9, 600.0), ((17, 16, 16), 2, 0, 20, 400.0), ((17, 16, 16), 2, 1, 9, 900.0),
         ((17, 16, 16), 1, 2, 31, 300.0), ((17, 16, 16), 1, 1, 60, 500.0), ((17, 16, 16), 2, 2, 1, 2000.0)]


@pytest.mark.parametrize("cells,elements,lanes,hot,speed", CASES)
def test_moved_atoms_match_the_oracle(built, beta_file, beta_file_2el, cells, elements, lanes, hot, speed):
    at = W.fcc_lattice(cells, seed=13)
    rng = np.random.default_rng(2)
    if elements == 2:
        at.type = np.where(rng.random(at.n) < 0.4, 2, 1).astype(np.int32)
        at.mass = np.array([0.0, W.NI_MASS, 55.845])
    hot_atoms(at, hot, speed, 4)
    words = W.fix_args(beta_file_2el if elements == 2 else beta_file, grid=(5, 4, 6), T_e=700.0,
                       elements=("Ni", "Fe")[:elements])
    gpu, ref = ephgb.FixEPH(words, at, dt=0.0005), OracleFix(words, at, 0.0005)
    if lanes:
        gpu.set_threads_per_atom(lanes)
    assert gpu.list_skin()[1]
    for s in range(8):
        stream = W.gaussian_stream(n_in_group(at), 9, s)
        gpu.step(1, xi=xi_rows(at, stream))
        ref.step(stream)
        for k in KEYS:
            err = key_err(k, gpu.get(k), ref.get(k))
            assert err <= TOL, (s, k, err)
