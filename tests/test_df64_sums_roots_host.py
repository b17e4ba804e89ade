"""The sum of four double-floats that the adjoint's coefficient gradients take
and the root that the EAM force sweep takes (df64::sum4 and sqrt_near,
user-eph_gb300/csrc/eph_df64.cuh), built for the host from the same source
(tests/native/df64_sum_check.cpp, df64_root_check.cpp).  No GPU.

Bound of the sum: seven FP64 additions in turn err by at most 3 + 2 + 1 rounding errors of
partial sums of up to 4 terms; one rounding of the sum, at most 4 terms large,
is 4 * 2^-53 of the largest, and what sum4 leaves out is far below that."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "user-eph_gb300", "csrc")


def test_sum_of_four_is_as_good_as_fp64(tmp_path):
    cxx = shutil.which(os.environ.get("CXX", "g++"))
    if not cxx:
        pytest.skip("no C++ compiler")
    exe = str(tmp_path / "df64_sum_check")
    subprocess.run([cxx, "-O2", "-ffp-contract=off", "-fno-fast-math", "-std=c++17", "-I" + CSRC, "-o", exe,
                    os.path.join(HERE, "native", "df64_sum_check.cpp")], check=True)
    worst, count = subprocess.run([exe], check=True, capture_output=True, text=True).stdout.split()
    assert int(count) == 2000000 and float(worst) <= 4.0


def test_root_of_the_pair_distance(tmp_path):
    """r of the EAM force sweep within 2^-47: the residual's roundings (2^-49 and
    2^-50 of the root), the square of the low part it leaves out (2^-49) and the
    rounding of the result's low part (2^-49)."""
    cxx = shutil.which(os.environ.get("CXX", "g++"))
    if not cxx:
        pytest.skip("no C++ compiler")
    exe = str(tmp_path / "df64_root_check")
    subprocess.run([cxx, "-O2", "-ffp-contract=off", "-fno-fast-math", "-std=c++17", "-I" + CSRC, "-o", exe,
                    os.path.join(HERE, "native", "df64_root_check.cpp")], check=True)
    assert float(subprocess.run([exe], check=True, capture_output=True, text=True).stdout) <= 1.0
