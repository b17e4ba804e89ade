"""Device memory of an adjoint on a grid past the cluster solve's size."""
import pytest

import ephgb
from ephgb import workloads as W
from ephgb.adjoint import Adjoint

pytestmark = pytest.mark.gpu


def test_large_grids_keep_only_the_recorded_substeps(built, beta_file):
    """Past the cluster's cells the reverse solve reads the recorded temperatures
    (8 B per substep and cell) and nothing else of that size is allocated."""
    torch = pytest.importorskip("torch")
    at = W.fcc_lattice(5, seed=3)
    g = (48, 48, 48)
    fix = ephgb.FixEPH(W.fix_args(beta_file, grid=g), at, dt=0.001)
    nsub, _ = ephgb.Grid(n=g, lo=at.boxlo, hi=at.boxhi).substeps(0.001)
    record = 8 * nsub * g[0] * g[1] * g[2]
    assert record > 1 << 30
    free = torch.cuda.mem_get_info()[0]
    adj = Adjoint(fix, checkpoint_every=1)
    adj.forward(1)
    assert free - torch.cuda.mem_get_info()[0] < 1.25 * record
