"""In-place FFT plans (gisspa_b200/csrc/planfft.cuh): factorisations on the CPU,
the kernel against a double DFT on a GPU (tests/native/test_planfft.cu)."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.mark.skipif(shutil.which("nvcc") is None, reason="nvcc not available")
@pytest.mark.parametrize("where", ["cpu", pytest.param("gpu", marks=pytest.mark.gpu)])
def test_planned_transforms(tmp_path, where):
    exe = str(tmp_path / "test_planfft")
    subprocess.run(["nvcc", "-std=c++17", "-O2", "--expt-relaxed-constexpr", "-gencode", "arch=compute_100a,code=sm_100a",
                    "-I" + os.path.join(ROOT, "gisspa_b200", "csrc"), "-o", exe,
                    os.path.join(ROOT, "tests", "native", "test_planfft.cu")], check=True)
    r = subprocess.run([exe, where], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr
    assert "OK" in r.stdout
