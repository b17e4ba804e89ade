"""eph_step (final_integrate and the deposits in one kernel, the force cleared by
initial_integrate) against the same step through the hooks, each its own
kernels: the same bits, whatever part of the fix is on."""
import numpy as np
import pytest

import ephgb
from ephgb import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", [ephgb.MODE_FAST, ephgb.MODE_EXACT])
@pytest.mark.parametrize("flags", [0, 1, 2, 3, 4, 5, 6, 7, 15])
def test_step_is_its_hooks(built, beta_file, mode, flags):
    at = W.fcc_lattice((5, 6, 5), seed=17)
    at.mask = np.where(np.arange(at.n) % 5 == 0, 2, 1).astype(np.int32)
    words = W.fix_args(beta_file, flags=flags, grid=(3, 4, 5), T_e=900.0)
    a, b = (ephgb.FixEPH(words, at, dt=0.001, mode=mode) for _ in range(2))
    f0 = np.random.default_rng(3).normal(0.0, 0.05, (at.n, 3))
    for fix in (a, b):
        fix.put("f", f0)
    for _ in range(3):
        a.step(1)
        b.initial_integrate()
        b.put("f", np.zeros((at.n, 3)))
        b.post_force()
        b.final_integrate()
        b.end_of_step()
    for k in ("x", "v", "f", "f_eph", "f_rng", "T"):
        assert np.array_equal(a.get(k), b.get(k)), k
    assert a.compute_vector(0) == b.compute_vector(0)
