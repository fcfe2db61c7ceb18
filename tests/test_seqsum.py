"""Float32 running sums in sequential order (gisspa_b200/csrc/seqsum.cuh)
against a plain loop of additions, bit for bit: the composition of runs on the
CPU, and the kernel on a GPU (tests/native/test_seqsum.cu)."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.mark.skipif(shutil.which("nvcc") is None, reason="nvcc not available")
@pytest.mark.parametrize("where", ["cpu", pytest.param("gpu", marks=pytest.mark.gpu)])
def test_running_sums_bit_for_bit(tmp_path, where):
    exe = str(tmp_path / "test_seqsum")
    subprocess.run(["nvcc", "-std=c++17", "-O2", "-gencode", "arch=compute_100a,code=sm_100a",
                    "-I" + os.path.join(ROOT, "gisspa_b200", "csrc"), "-o", exe,
                    os.path.join(ROOT, "tests", "native", "test_seqsum.cu")], check=True)
    r = subprocess.run([exe, where], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout + r.stderr
    assert "OK" in r.stdout
