"""Row and bin capacities of the kept lists where the box's mean density says
little of an atom's surroundings: what fits a bin search every step fits the
lists, which reach farther and use wider bins.  Against that search, at the bars
of tests/test_gpu_eam_lists.py."""
import numpy as np
import pytest

import ephgb
from ephgb import workloads as W
from test_gpu_eam_lists import agree, ni_eam

pytestmark = pytest.mark.gpu


def compare(got, ref, n, steps=2, seed=12):
    rng = np.random.default_rng(seed)
    for _ in range(steps):
        xi = rng.standard_normal((n, 3))
        for f in (got, ref):
            f.step(1, xi=xi)
        agree(got, ref)


# cells, the box along z in crystals, pair force, the fix's cut-off, the user's
# bin capacity: a third full; a fifth full, the next lattice shell just outside
# the cut-off; a full box and a capacity of the caller's
BOXES = [((17, 16, 17), 3.0, True, 4.6, 0), ((19, 16, 18), 3.0, True, 4.6, 0), ((17, 16, 17), 5.0, False, 4.9, 0),
         ((17, 16, 17), 1.0, False, 4.9, 16)]


@pytest.mark.parametrize("cells,stretch,eam,cutoff,bins", BOXES)
def test_lists_take_what_a_search_takes(built, tmp_path, cells, stretch, eam, cutoff, bins):
    at = W.fcc_lattice(cells, seed=62, jitter=0.02)
    at.boxhi = at.boxhi * np.array([1.0, 1.0, stretch])
    words = W.fix_args(W.write_beta_file(str(tmp_path / "f.beta"), rc=cutoff), grid=(9, 8, 10), T_e=900.0)
    pair = (ni_eam(tmp_path), ["Ni"]) if eam else None
    got, ref = (ephgb.FixEPH(words, dt=0.0005, mass=at.mass, boxlo=at.boxlo, boxhi=at.boxhi, eam=pair) for _ in range(2))
    for f, skin in ((got, 0.3), (ref, 0.0)):
        if bins:
            f.set_capacity(bins=bins)
        f.set_list_skin(skin)
        f.set_atoms(at.x, at.v, at.type, at.mask)
    assert got.list_skin()[1] and not ref.list_skin()[1]
    compare(got, ref, at.n)


@pytest.mark.parametrize("change", [dict(bins=48), dict(pairs=112), dict(bins=40, pairs=120)])
def test_a_new_capacity_starts_new_lists(built, beta_file, change):
    """eph_set_capacity gives the bins that the lists and moved atoms read anew."""
    at = W.fcc_lattice((17, 16, 17), seed=62)
    at.v[::1500] *= 300.0  # a few atoms that move between builds
    words = W.fix_args(beta_file, grid=(9, 8, 10), T_e=900.0)
    got, ref = (ephgb.FixEPH(words, at, dt=0.0005) for _ in range(2))
    got.set_list_skin(0.3)
    ref.set_list_skin(0.0)
    compare(got, ref, at.n)
    builds = got.counter("build")
    got.set_capacity(**change)
    compare(got, ref, at.n, seed=13)
    assert got.counter("build") == builds + 1


@pytest.mark.parametrize("skin", [0.0, 0.3])
def test_more_pairs_than_rows_is_an_error(built, beta_file, tmp_path, skin):
    """A fifth of the box full: 80 pair rows for 85 to 91 pairs of the pair force
    (and room for their candidates in the lists).  An error, every step, and the
    context still answers."""
    at = W.fcc_lattice((17, 16, 17), seed=62, jitter=0.02)
    at.boxhi = at.boxhi * np.array([1.0, 1.0, 5.0])
    fix = ephgb.FixEPH(W.fix_args(beta_file, grid=(9, 8, 10)), at, dt=0.0005, eam=(ni_eam(tmp_path), ["Ni"]))
    fix.set_list_skin(skin)
    for _ in range(2):
        fix.step(1)
        with pytest.raises(ephgb.EphError) as e:
            fix.synchronize()
        assert e.value.status == 4  # EPH_ERR_CAPACITY
    assert fix.get("T").size == 720
