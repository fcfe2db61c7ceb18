"""A bounded wait of the persistent correlation that gives up: flag and NaN
scores (tests/native/test_corr_timeout.cu)."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

pytestmark = pytest.mark.gpu


def test_wait_that_gives_up_scores_nan(tmp_path):
    exe = str(tmp_path / "test_corr_timeout")
    subprocess.run(["nvcc", "-std=c++17", "-O2", "--expt-relaxed-constexpr", "-gencode", "arch=compute_100a,code=sm_100a",
                    "-I" + os.path.join(ROOT, "gisspa_b200", "csrc"), "-o", exe,
                    os.path.join(ROOT, "tests", "native", "test_corr_timeout.cu")], check=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout + r.stderr
    assert "OK" in r.stdout
