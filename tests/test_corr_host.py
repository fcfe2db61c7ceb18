"""Host-compiled parts of the persistent correlation (tests/native/test_corr_host.cu)."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def exe(tmp_path_factory):
    if shutil.which("nvcc") is None:
        pytest.skip("nvcc not available")
    out = str(tmp_path_factory.mktemp("corr_host") / "test_corr_host")
    subprocess.run(["nvcc", "-std=c++17", "-O1", "--expt-relaxed-constexpr",
                    "-gencode", "arch=compute_100a,code=sm_100a", "-diag-suppress", "177",
                    "-I" + os.path.join(ROOT, "gisspa_b200", "csrc"), "-o", out,
                    os.path.join(ROOT, "tests", "native", "test_corr_host.cu")], check=True)
    return out


@pytest.mark.parametrize("what", ["claims", "border", "rings"])
def test_corr_host(exe, what):
    r = subprocess.run([exe, what], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr
    assert "OK" in r.stdout
