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
         ("eam", (17, 16, 17), 1), ("eam", (25, 24, 26), 1), ("eam", (37, 38, 36), 1),
         ("eamlist", (17, 16, 17), 1), ("eamlist", (25, 24, 26), 1), ("eamlist", (45, 46, 47), 1)]


@pytest.mark.parametrize("source,cells,elements", CASES)
def test_lanes_and_sources_match_fp64(built, beta_file, beta_file_2el, tmp_path, source, cells, elements):
    words, at = system(cells, beta_file_2el if elements == 2 else beta_file, elements, source.startswith("eam"))
    eam = None
    if source.startswith("eam"):
        path = str(tmp_path / "Ni.eam")
        with open(NI_EAM, "rb") as src, open(path, "wb") as dst:
            dst.write(lzma.decompress(src.read()))
        eam = (path, ["Ni"])
    got, ref = (ephgb.FixEPH(words, at, dt=0.0005, eam=eam) for _ in range(2))
    got.set_list_skin(0.3 if source.endswith("list") else 0.0)
    ref.set_list_skin(0.0)
    ref.set_pair_arithmetic(ephgb.PAIRS_FP64)
    assert got.list_skin()[1] == source.endswith("list")
    rng = np.random.default_rng(11)
    for _ in range(3):
        xi = rng.standard_normal((at.n, 3))
        for f in (got, ref):
            f.step(1, xi=xi)
        # the EAM force is the larger part of f and runs in either arithmetic
        for k in KEYS:
            if source.startswith("eam") and k in ("x", "v", "f", "w", "f_eph"):
                tol = 1e-11  # EAM bar (tests/test_gpu_eam.py)
            else:
                tol = TOL
            err = atom_err(got.get(k), ref.get(k))
            assert err <= tol, (k, err)


def write_two_element_setfl(path, nr=2001, nrho=1501, rc=5.6, rho_max=120.0):
    """A setfl file of two made-up elements (smooth tables that differ)."""
    dr, drho = rc / (nr - 1), rho_max / (nrho - 1)
    r, rho = np.arange(nr) * dr, np.arange(nrho) * drho
    cut = np.clip(1.0 - r / rc, 0.0, None) ** 3
    with open(path, "w") as f:
        f.write(f"#\n#\n#\n2 Ni Xx\n{nrho} {drho!r} {nr} {dr!r} {rc!r}\n")
        for k, (a, b) in enumerate(((1.0, 9.0), (1.4, 7.0))):
            f.write(f"{28 + k} 58.69 3.52 fcc\n")
            for arr in (-a * np.sqrt(rho + 0.1), b * np.exp(-0.5 * r) * cut):
                f.write("\n".join(repr(float(v)) for v in arr) + "\n")
        for s in (4.0, 3.0, 5.0):  # 11, 21, 22
            f.write("\n".join(repr(float(v)) for v in s * np.exp(-1.1 * r) * cut * r) + "\n")
    return path


@pytest.mark.parametrize("skin", [0.0, 0.3])
def test_two_element_pair_force_matches_the_restatement(built, beta_file, tmp_path, skin):
    """Pairs of unlike setfl elements (f_a and f_b tables apart), over the bins
    and over kept lists, against the numpy restatement at the bar of
    tests/test_gpu_eam.py (energy 1e-12, forces 1e-11)."""
    from oracle.eam_ref import energy_forces, read_setfl

    at = W.fcc_lattice((6, 6, 6), seed=81)
    at.type = np.where(np.random.default_rng(2).random(at.n) < 0.4, 2, 1).astype(np.int32)
    at.mass = np.array([0.0, W.NI_MASS, W.NI_MASS])
    path = write_two_element_setfl(str(tmp_path / "two.eam"))
    fix = ephgb.FixEPH(W.fix_args(beta_file, flags=9, grid=(4, 4, 4), elements=("Ni", "Ni")), at, dt=0.001,
                       eam=(path, ["Ni", "Xx"]))
    if skin:
        fix.set_threads_per_atom(1)
    fix.set_list_skin(skin)
    assert fix.list_skin()[1] == (skin > 0)
    E, f = energy_forces(read_setfl(path), at.x, at.type, {1: 0, 2: 1}, at.boxhi - at.boxlo)
    for _ in range(2):  # flags 9: friction on, no integration: x stays
        fix.step(1)
        got = fix.get("f") - fix.get("f_eph")
        assert abs(fix.pair_energy() - E) <= 1e-12 * abs(E)
        assert np.abs(got - f).max() <= 1e-11 * np.abs(f).max()
