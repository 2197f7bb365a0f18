"""The spatial order's curve and the finest cut of the mixed pair work, checked
on the host: a host program built with nvcc, no GPU needed."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_hilbert_curve_and_finest_cut(tmp_path):
    nvcc = shutil.which("nvcc") or ("/usr/local/cuda/bin/nvcc" if os.path.exists("/usr/local/cuda/bin/nvcc") else None)
    if nvcc is None:
        pytest.skip("nvcc not available")
    exe = str(tmp_path / "host_rules")
    cmd = [nvcc, "-std=c++17", "-O1", "-I", os.path.join(ROOT, "nbodygo_gb300", "csrc"), "-I",
           os.path.join(ROOT, "include"), os.path.join(ROOT, "tests", "cpp", "host_rules.cu"), "-o", exe]
    r = subprocess.run(cmd, capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    r = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0 and "hilbert bad 0, cut bad 0" in r.stdout, r.stdout + r.stderr
