"""The order of copies and kernels over streams, read from a CUDA runtime that
only logs its calls (tests/native/cudart_log.cpp).  No GPU."""
import os
import shutil
import subprocess
import sys

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
PKG = os.path.join(os.path.dirname(HERE), "user-eph_gb300")


@pytest.fixture(scope="module")
def logged(built, tmp_path_factory):
    """Runs a program with the logging runtime; its log, as lists of words."""
    cxx = shutil.which(os.environ.get("CXX", "g++"))
    if not cxx:
        pytest.skip("no C++ compiler")
    lib = str(tmp_path_factory.mktemp("cudart") / "cudart_log.so")
    subprocess.run([cxx, "-O1", "-shared", "-fPIC", "-std=c++17", "-o", lib, os.path.join(HERE, "native", "cudart_log.cpp")],
                   check=True)

    def run(program):
        env = dict(os.environ, LD_PRELOAD=lib, PYTHONPATH=os.pathsep.join([PKG, HERE]))
        out = subprocess.run([sys.executable, "-c", program], env=env, capture_output=True, text=True)
        assert out.returncode == 0, out.stderr[-2000:]
        return [line.split(None, 2) for line in out.stderr.splitlines() if line.split()[:1][0] in ("default", "stream", "wait", "mark")]

    return run


def test_set_up_copies_are_ordered_with_the_kernels(logged, beta_file, tmp_path):
    """Nothing orders the default stream with a context's: grid arrays,
    tables, atoms and parameters are copied on the context's own, the grid's
    coefficients are made after them."""
    log = logged(f"""
import sys
import numpy as np
import ephgb
from ephgb import workloads as W
from ephgb.adjoint import Adjoint
at = W.fcc_lattice(6)
grid = W.write_grid_file({str(tmp_path / "T.in")!r})
pair = W.write_eam_sutton_chen({str(tmp_path / "Ni.eam")!r})
ephgb.FixEPH(W.fix_args({beta_file!r}, T_infile=grid), at, eam=(pair, ["Ni"])).step(1)
fix = ephgb.FixEPH(W.fix_args({beta_file!r}), at)
Adjoint(fix, checkpoint_every=2)
fix.set_beta_knots(0, np.linspace(1.0, 0.0, 2000), np.full(2000, 0.05))
fix.set_grid_constants(3e-6, 0.2)
fix.step(1)
""")
    assert sum("k_fdm_coef" in words[-1] for words in log) == 1
    assert [words for words in log if words[0] == "default"] == []


@pytest.mark.parametrize("change", ["reset_dt(0.0005)", "set_grid_constants(3e-6, 0.2)",
                                    "set_beta_knots(0, np.linspace(1.0, 0.0, 2000), np.full(2000, 0.05))"])
def test_a_replica_changes_after_the_queued_steps(logged, beta_file, change):
    """A batch's steps run on its own stream: a replica's new time step, grid
    constants or tables wait for those queued before."""
    log = logged(f"""
import numpy as np
import sys
import ephgb
from ephgb import workloads as W
at = W.fcc_lattice(5)
batch = ephgb.Batch([(W.fix_args({beta_file!r}), at)] * 2)
batch.step(3)
fix = batch.replicas[1]
sys.stderr.write("mark change\\n")
fix.{change}
""")
    last = max(i for i, words in enumerate(log) if words[-1] == "cudaGraphLaunch")
    stream = log[last][1]
    after = log[log.index(["mark", "change"]):]
    first_work = next(i for i, words in enumerate(after) if words[0] in ("stream", "default"))
    assert ["wait", stream] in after[:first_work]
