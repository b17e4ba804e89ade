"""The df64 sweeps at the sizes where their lanes per atom change (1, 2 and 4),
over each source of candidates (bin search, kept lists, the EAM engine's pair
list), against the FP64 pair arithmetic with a bin search every step: two
elements, atoms outside the group, a fast knock-on atom (moved atoms, wraps,
images across the box faces) and box edges that differ.

Tolerance: both arithmetics hold the 1e-12 bar against the reference per atom
(tests/test_gpu_parity.py), so they differ by at most 2e-12."""
import lzma
import os

import numpy as np
import pytest

import ephgb
from ephgb import workloads as W
from helpers import atom_err

pytestmark = pytest.mark.gpu
TOL = 2e-12
KEYS = ("rho", "w", "f_eph", "f_rng", "f", "x", "v", "T")
NI_EAM = os.path.join(os.path.dirname(__file__), "golden", "ref_inputs", "MD_Run_Ni.eam.xz")


def system(cells, beta_file, elements, eam=False):
    at = W.fcc_lattice(cells, seed=61)
    rng = np.random.default_rng(3)
    if elements == 2:
        at.type = np.where(rng.random(at.n) < 0.4, 2, 1).astype(np.int32)
        at.mass = np.array([0.0, W.NI_MASS, 55.845])
    if not eam:
        at.mask = np.where(rng.random(at.n) < 0.1, 2, 1).astype(np.int32)
    # a 10 keV atom about to cross three box faces
    at.x[7] = at.boxhi - np.array([0.4, 0.3, 0.2])
    at.v[7] = np.array([1000.0, 1100.0, 900.0])
    return W.fix_args(beta_file, grid=(9, 8, 10), T_e=900.0, elements=("Ni", "Fe")[:elements]), at


# lanes 4, 2, 1 of each source (the smallest and largest sides of each rule
# that stay quick), odd atom counts so that last blocks are partial
CASES = [("list", (17, 16, 17), 2), ("list", (25, 24, 26), 1), ("list", (33, 32, 31), 2),
         ("bins", (17, 16, 17), 1), ("bins", (25, 24, 26), 2), ("bins", (43, 44, 42), 1),
         ("eam", (17, 16, 17), 1), ("eam", (25, 24, 26), 1), ("eam", (37, 38, 36), 1)]


@pytest.mark.parametrize("source,cells,elements", CASES)
def test_lanes_and_sources_match_fp64(built, beta_file, beta_file_2el, tmp_path, source, cells, elements):
    words, at = system(cells, beta_file_2el if elements == 2 else beta_file, elements, source == "eam")
    eam = None
    if source == "eam":
        path = str(tmp_path / "Ni.eam")
        with open(NI_EAM, "rb") as src, open(path, "wb") as dst:
            dst.write(lzma.decompress(src.read()))
        eam = (path, ["Ni"])
    got, ref = (ephgb.FixEPH(words, at, dt=0.0005, eam=eam) for _ in range(2))
    got.set_list_skin(0.3 if source == "list" else 0.0)
    ref.set_list_skin(0.0)
    ref.set_pair_arithmetic(ephgb.PAIRS_FP64)
    assert got.list_skin()[1] == (source == "list")
    rng = np.random.default_rng(11)
    for _ in range(3):
        xi = rng.standard_normal((at.n, 3))
        for f in (got, ref):
            f.step(1, xi=xi)
        # the EAM force is the larger part of f and runs in either arithmetic
        for k in KEYS:
            if source == "eam" and k in ("x", "v", "f", "w", "f_eph"):
                tol = 1e-11  # EAM bar (tests/test_gpu_eam.py)
            else:
                tol = TOL
            err = atom_err(got.get(k), ref.get(k))
            assert err <= tol, (k, err)
