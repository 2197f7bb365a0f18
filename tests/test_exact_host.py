"""nbg_exact.h (correctly rounded products, quotients and roots from integers)
against the host's IEEE operations: a host program, no GPU needed."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.mark.parametrize("seed", [1, 2])
def test_exact_arithmetic_matches_ieee(tmp_path, seed):
    nvcc = shutil.which("nvcc") or ("/usr/local/cuda/bin/nvcc" if os.path.exists("/usr/local/cuda/bin/nvcc") else None)
    if nvcc is None:
        pytest.skip("nvcc not available")
    exe = str(tmp_path / "exact_host")
    cmd = [nvcc, "-std=c++17", "-O2", "-Xcompiler", "-ffp-contract=off", "-I",
           os.path.join(ROOT, "nbodygo_gb300", "csrc"), os.path.join(ROOT, "tests", "cpp", "exact_host.cu"), "-o", exe]
    r = subprocess.run(cmd, capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    r = subprocess.run([exe, "4000000", str(seed)], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0 and ", bad 0" in r.stdout, r.stdout + r.stderr
