"""The margin of the FP64 division and square root on the integer pipes
(fc3dgpu_ieee64.cuh): right on the host with seeds off by up to 3 units in the
last place, and on the device, where the approximate instructions' errors (at
most 1 unit for the reciprocal, 2^-22.9 or 2.1 units for the reciprocal root) stay
within it and zeros, subnormals, infinities and NaN take the compiler's form."""
import subprocess

import pytest

from test_ieee64 import CSRC, HERE, checker  # noqa: F401


@pytest.mark.parametrize("ulps", [-3, 3])
def test_seeds_off_by_three_units(checker, ulps):  # noqa: F811
    out = subprocess.run([str(checker), str(ulps), "1000000"], check=True, capture_output=True, text=True)
    assert out.stdout.strip() == "0"


@pytest.mark.gpu
def test_device(tmp_path):
    from siconos_gb300 import build as B
    exe = tmp_path / "check"
    subprocess.run([B._nvcc(), "-gencode", "arch=compute_103a,code=sm_103a", "-O3", "-std=c++17", "--fmad=false",
                    f"-I{CSRC}", "-o", str(exe), str(HERE / "ieee64_device_check.cu")], check=True)
    bad, rcp, rsqrt = subprocess.run([str(exe)], check=True, capture_output=True, text=True, timeout=120).stdout.split()
    assert bad == "0"
    assert float(rcp) <= 3.0 and float(rsqrt) <= 3.0
