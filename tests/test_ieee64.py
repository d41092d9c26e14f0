"""The FP64 division, square root and comparisons that the kernels form on the
integer pipes (fc3dgpu_ieee64.cuh), compiled for the host: the same bits as the
compiler's for every operand, whatever the seeds' errors up to 2 units in the
last place (the hardware approximations' is 1)."""
import shutil
import subprocess
from pathlib import Path

import pytest

HERE = Path(__file__).resolve().parent
CSRC = HERE.parent / "siconos_gb300" / "csrc"


@pytest.fixture(scope="module")
def checker(tmp_path_factory):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    inc = Path(nvcc).resolve().parent.parent / "include"
    exe = tmp_path_factory.mktemp("ieee64") / "check"
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", f"-I{CSRC}", f"-I{inc}", "-o", str(exe),
                    str(HERE / "ieee64_check.cpp")], check=True)
    return exe


@pytest.mark.parametrize("ulps", [-2, -1, 0, 1, 2])
def test_same_bits_as_the_compiler(checker, ulps):
    out = subprocess.run([str(checker), str(ulps), "1000000"], check=True, capture_output=True, text=True)
    assert out.stdout.strip() == "0"
