"""The Barnes-Hut tree's octant paths from grid cells against the descent,
bit for bit, by a host program built with nvcc: no GPU needed."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_cells_give_the_descents_path(tmp_path):
    nvcc = shutil.which("nvcc") or ("/usr/local/cuda/bin/nvcc" if os.path.exists("/usr/local/cuda/bin/nvcc") else None)
    if nvcc is None:
        pytest.skip("nvcc not available")
    exe = str(tmp_path / "octant_host")
    cmd = [nvcc, "-std=c++17", "-O1", "-Xcompiler", "-ffp-contract=off", "-I",
           os.path.join(ROOT, "nbodygo_gb300", "csrc"), os.path.join(ROOT, "tests", "cpp", "octant_host.cu"), "-o", exe]
    r = subprocess.run(cmd, capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    r = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0 and "octant bad 0" in r.stdout, r.stdout + r.stderr
