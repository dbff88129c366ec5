"""The packed reciprocal of the shifted forms rounds as the division does."""
import os
import shutil
import subprocess

import pytest

pytestmark = pytest.mark.gpu

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "latticeboltzmannmethod-fonnesu-grassi-guffanti_b200", "csrc")


def test_inverse_mid_equals_the_division_for_every_pattern(tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("no nvcc")
    exe = str(tmp_path / "reciprocal")
    subprocess.check_call([nvcc, "-gencode", "arch=compute_100a,code=sm_100a", "-std=c++17", "-O3", "--fmad=false", "-I",
                           CSRC, "-o", exe, os.path.join(HERE, "native", "reciprocal.cu")])
    out = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert out.returncode == 0, out.stderr
    mids, differ, guard = map(int, out.stdout.split())
    # both ends exclusive: 240 binades of 2^23 values less the lower end itself
    assert mids == 240 * 2**23 - 1
    assert differ == 0 and guard == 0
