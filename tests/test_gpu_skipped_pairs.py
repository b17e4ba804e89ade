"""Neighbours the reference skips (outside the group) in the FAST force sweeps:
from none to nearly all of an atom's, one and two elements, in the FP64 and the
df64 sweeps and at each count of lanes, against the oracle (1e-12 per atom, the
parity tests' bar)."""
import numpy as np
import pytest

import ephgb
from ephgb import workloads as W
from helpers import key_err, n_in_group, xi_rows
from oracle.bindings import OracleFix

pytestmark = pytest.mark.gpu
TOL = 1e-12
CASES = [((6, 5, 5), 1, 0.02, 8), ((6, 5, 5), 2, 0.5, 4), ((6, 5, 5), 2, 0.97, 1), ((6, 5, 5), 1, 0.9, 2),
         ((16, 16, 17), 1, 0.3, 1), ((16, 16, 17), 2, 0.3, 4), ((16, 16, 17), 2, 0.95, 2), ((16, 16, 17), 1, 0.05, 8)]


@pytest.mark.parametrize("flags", [7, 5])
@pytest.mark.parametrize("cells,elements,outside,lanes", CASES)
def test_skipped_pairs_match_the_oracle(built, beta_file, beta_file_2el, cells, elements, outside, lanes, flags):
    at = W.fcc_lattice(cells, seed=23)
    rng = np.random.default_rng(8)
    if elements == 2:
        at.type = np.where(rng.random(at.n) < 0.4, 2, 1).astype(np.int32)
        at.mass = np.array([0.0, W.NI_MASS, 55.845])
    at.mask = np.where(rng.random(at.n) < outside, 2, 1).astype(np.int32)
    words = W.fix_args(beta_file_2el if elements == 2 else beta_file, flags=flags, grid=(5, 4, 6), T_e=700.0,
                       elements=("Ni", "Fe")[:elements])
    gpu, ref = ephgb.FixEPH(words, at, dt=0.001), OracleFix(words, at, 0.001)
    gpu.set_threads_per_atom(lanes)
    for s in range(2):
        stream = W.gaussian_stream(n_in_group(at), 9, s) if flags & 2 else None
        gpu.step(1, xi=xi_rows(at, stream)) if flags & 2 else gpu.step(1)
        ref.step(stream)
        for k in ("rho", "w", "f_eph", "f_rng", "f", "x", "v"):
            err = key_err(k, gpu.get(k), ref.get(k))
            assert err <= TOL, (s, k, err)
