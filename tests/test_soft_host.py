"""The FP64 products and quotients on the integer units
(user-eph_gb300/csrc/eph_softfp.cuh), built for the host from the same source:
every bit of 20 million products and quotients (tests/native/soft_check.cpp).
No GPU."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "user-eph_gb300", "csrc")


def test_products_and_quotients_bit_for_bit(tmp_path):
    cxx = shutil.which(os.environ.get("CXX", "g++"))
    if not cxx:
        pytest.skip("no C++ compiler")
    exe = str(tmp_path / "soft_check")
    subprocess.run([cxx, "-O2", "-ffp-contract=off", "-fno-fast-math", "-std=c++17", "-I" + CSRC, "-o", exe,
                    os.path.join(HERE, "native", "soft_check.cpp")], check=True)
    out = subprocess.run([exe], check=True, capture_output=True, text=True).stdout
    assert out.split() == ["mul", "0", "div", "0"]
