"""Transforms of the windows l = 16 N2 on the CPU (tests/native/test_winfft.cu)."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.mark.skipif(shutil.which("nvcc") is None, reason="nvcc not available")
def test_window_transforms_against_double_dft(tmp_path):
    exe = str(tmp_path / "test_winfft")
    subprocess.run(["nvcc", "-std=c++17", "-O1", "--expt-relaxed-constexpr",
                    "-gencode", "arch=compute_100a,code=sm_100a", "-diag-suppress", "177",
                    "-I" + os.path.join(ROOT, "gisspa_b200", "csrc"), "-o", exe,
                    os.path.join(ROOT, "tests", "native", "test_winfft.cu")], check=True)
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr
    assert "OK" in r.stdout
