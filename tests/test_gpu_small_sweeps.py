"""The small-system density sweep (k_density_tpa) at the sizes where its lanes
per atom change (32, 16, 8, 4, and 2 on request) against the oracle: one and
two elements, part of the atoms outside the group, friction on and off (the
sums of M_i and S_i, or rho_i alone), uneven boxes.  The bar is the parity
tests' 1e-12 per atom."""
import numpy as np
import pytest

import ephgb
from ephgb import workloads as W
from helpers import key_err, n_in_group, xi_rows
from oracle.bindings import OracleFix

pytestmark = pytest.mark.gpu
TOL = 1e-12
KEYS = ("rho", "w", "f_eph", "f_rng", "f", "x", "v", "array", "T")

# cells (4 atoms each), elements, flags, lanes asked for (0: the rule)
CASES = [((5, 5, 5), 1, 7, 0), ((7, 7, 7), 2, 7, 0), ((8, 7, 9), 1, 6, 0), ((11, 11, 11), 2, 7, 0),
         ((12, 11, 13), 1, 7, 0), ((14, 15, 14), 2, 6, 0), ((15, 14, 16), 1, 7, 0), ((5, 6, 7), 2, 7, 2),
         ((5, 6, 7), 1, 7, 4), ((6, 5, 7), 1, 7, 8)]


@pytest.mark.parametrize("cells,elements,flags,lanes", CASES)
def test_small_sweeps_match_the_oracle(built, beta_file, beta_file_2el, cells, elements, flags, lanes):
    at = W.fcc_lattice(cells, seed=71)
    rng = np.random.default_rng(5)
    if elements == 2:
        at.type = np.where(rng.random(at.n) < 0.4, 2, 1).astype(np.int32)
        at.mass = np.array([0.0, W.NI_MASS, 55.845])
    at.mask = np.where(rng.random(at.n) < 0.1, 2, 1).astype(np.int32)
    words = W.fix_args(beta_file_2el if elements == 2 else beta_file, flags=flags, grid=(5, 4, 6), T_e=700.0,
                       elements=("Ni", "Fe")[:elements])
    gpu, ref = ephgb.FixEPH(words, at, dt=0.001), OracleFix(words, at, 0.001)
    if lanes:
        gpu.set_threads_per_atom(lanes)
    for s in range(2):
        stream = W.gaussian_stream(n_in_group(at), 9, s)
        gpu.step(1, xi=xi_rows(at, stream))
        ref.step(stream)
        for k in KEYS:
            err = key_err(k, gpu.get(k), ref.get(k))
            assert err <= TOL, (s, k, err)
