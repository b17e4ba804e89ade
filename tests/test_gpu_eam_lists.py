"""Kept candidate lists that the EAM engine's pair force shares with the fix's
density sweep, against a bin search every step (list skin 0, or FP64 pair terms).

Tolerance: the bars of tests/test_gpu_eam.py, forces 1e-11 and energy 1e-12;
rho 2e-12 (either arithmetic is within 1e-12 of the reference)."""
import lzma
import os

import numpy as np
import pytest

import ephgb
from ephgb import workloads as W
from helpers import atom_err

pytestmark = pytest.mark.gpu
NI_EAM = os.path.join(os.path.dirname(__file__), "golden", "ref_inputs", "MD_Run_Ni.eam.xz")


def ni_eam(folder):
    path = str(folder / "Ni.eam")
    with open(NI_EAM, "rb") as src, open(path, "wb") as dst:
        dst.write(lzma.decompress(src.read()))
    return path


def agree(got, ref):
    for k in ("rho", "x", "v", "f"):
        err = atom_err(got.get(k), ref.get(k))
        assert err <= (2e-12 if k == "rho" else 1e-11), (k, err)
    E = ref.pair_energy()
    assert abs(got.pair_energy() - E) <= 1e-12 * abs(E)


def with_and_without_lists(words, at, eam, skin=0.3):
    got, ref = (ephgb.FixEPH(words, at, dt=0.0005, eam=(eam, ["Ni"])) for _ in range(2))
    got.set_list_skin(skin)
    ref.set_list_skin(0.0)
    assert got.list_skin()[1] and not ref.list_skin()[1]
    return got, ref


@pytest.mark.parametrize("builder", ["shorter pair cut-off", "hook"])
def test_atoms_outside_the_group_keep_their_lists(built, beta_file, tmp_path, builder):
    """A build made by the fix's sweep -- where the EAM list does not hold its
    pairs, or in post_force by itself -- leaves the pair force's lists whole."""
    at = W.fcc_lattice((17, 16, 17), seed=61)
    at.mask = np.where(np.random.default_rng(5).random(at.n) < 0.3, 2, 1).astype(np.int32)
    words = W.fix_args(beta_file, grid=(9, 8, 10), T_e=900.0)  # the fix's cut-off is 4.6 A
    if builder == "hook":
        eam = ni_eam(tmp_path)
    else:
        eam = W.write_eam_sutton_chen(str(tmp_path / "short.eam"), rc=4.4, r_on=3.6)
    got, ref = with_and_without_lists(words, at, eam)
    rng = np.random.default_rng(11)
    if builder == "hook":
        xi = rng.standard_normal((at.n, 3))
        for f in (got, ref):
            f.post_force(xi)
    for _ in range(3):
        xi = rng.standard_normal((at.n, 3))
        for f in (got, ref):
            f.step(1, xi=xi)
        agree(got, ref)


def hot_atoms(at, count, speed, seed):
    rng = np.random.default_rng(seed)
    hot = rng.choice(at.n, count, replace=False)
    u = rng.standard_normal((count, 3))
    at.v[hot] = speed * u / np.sqrt((u * u).sum(1))[:, None]


# 8 and 4 lanes per atom; half the box empty (the row capacities, which follow
# the box's mean density, are then those of half the atoms' neighbours); pair
# forces longer and shorter than the fix's cut-off; a skin that puts more
# candidates than rows around an atom
MOVED = [((17, 16, 17), 2.0, "ni", 0.3), ((21, 20, 20), 2.0, "ni", 0.3), ((17, 16, 17), 1.0, "short", 0.6),
         ((17, 16, 17), 1.0, "ni", 2.0), ((17, 16, 17), 1.0, "hook", 0.3)]


@pytest.mark.parametrize("cells,stretch,eam,skin", MOVED)
def test_moved_atoms_find_every_neighbour(built, beta_file, tmp_path, cells, stretch, eam, skin):
    at = W.fcc_lattice(cells, seed=62)
    at.boxhi = at.boxhi * np.array([1.0, 1.0, stretch])
    hot_atoms(at, 12, 900.0 if skin < 1.0 else 2200.0, 3)
    words = W.fix_args(beta_file, grid=(9, 8, 10), T_e=900.0)
    path = W.write_eam_sutton_chen(str(tmp_path / "short.eam"), rc=2.7, r_on=2.55) if eam == "short" else ni_eam(tmp_path)
    got, ref = with_and_without_lists(words, at, path, skin)
    rng = np.random.default_rng(12)
    builds = []
    for _ in range(4):
        xi = rng.standard_normal((at.n, 3))
        for f in (got, ref):
            f.step(1, xi=xi)
            if eam == "hook":
                f.post_force(xi)
        agree(got, ref)
        builds.append(got.counter("build"))
    assert builds[-1] == builds[0]  # the atoms moved between builds


@pytest.mark.parametrize("cells", [(17, 16, 17), (21, 20, 20)])
def test_two_elements_over_lists(built, beta_file, tmp_path, cells):
    """Unlike pairs (f_a and f_b tables apart) at 8 and 4 lanes per atom, against
    FP64 pair terms and a search every step."""
    from test_gpu_df_sweeps import write_two_element_setfl

    at = W.fcc_lattice(cells, seed=63)
    at.type = np.where(np.random.default_rng(2).random(at.n) < 0.4, 2, 1).astype(np.int32)
    at.mass = np.array([0.0, W.NI_MASS, W.NI_MASS])
    hot_atoms(at, 6, 700.0, 3)
    words = W.fix_args(beta_file, grid=(9, 8, 10), T_e=900.0, elements=("Ni", "Ni"))
    pair = (write_two_element_setfl(str(tmp_path / "two.eam")), ["Ni", "Xx"])
    got, ref = (ephgb.FixEPH(words, at, dt=0.0005, eam=pair) for _ in range(2))
    assert got.list_skin()[1]
    ref.set_pair_arithmetic(ephgb.PAIRS_FP64)
    assert not ref.list_skin()[1]
    rng = np.random.default_rng(13)
    for _ in range(3):
        xi = rng.standard_normal((at.n, 3))
        for f in (got, ref):
            f.step(1, xi=xi)
        agree(got, ref)
