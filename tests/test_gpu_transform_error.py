"""Rounding of the transforms' twiddles (tests/native)."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("name", ["test_fft16_error", "test_plan_twiddles"])
def test_transform_error(tmp_path, name):
    exe = str(tmp_path / name)
    subprocess.run(["nvcc", "-std=c++17", "-O2", "--expt-relaxed-constexpr", "-gencode", "arch=compute_100a,code=sm_100a",
                    "-I" + os.path.join(ROOT, "gisspa_b200", "csrc"), "-o", exe,
                    os.path.join(ROOT, "tests", "native", name + ".cu")], check=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout + r.stderr
    assert "OK" in r.stdout
