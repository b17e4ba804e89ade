"""FP64 products and quotients on the integer units, as the device computes
them (the host's half is tests/test_soft_host.py): every bit of 400 million
products and quotients, over every seed of the reciprocal
(tests/native/soft_device_check.cu)."""
import os
import subprocess

import pytest

from ephgb import build

pytestmark = pytest.mark.gpu
HERE = os.path.dirname(os.path.abspath(__file__))


def test_products_and_quotients_on_the_device(tmp_path):
    exe = str(tmp_path / "soft_device_check")
    subprocess.run([build.NVCC] + build.ARCH + ["-O3", "-fmad=false", "-std=c++17", "-I" + build.CSRC, "-o", exe,
                    os.path.join(HERE, "native", "soft_device_check.cu")], check=True)
    out = subprocess.run([exe], check=True, capture_output=True, text=True, timeout=120).stdout
    assert out.split() == ["mul", "0", "div", "0"]
