"""The shape a mixed context takes when it is given none: the rule on the host
(a program built with nvcc, no GPU needed), and on the GPU that the rule's
shape is the one that runs, bit for bit, and that a set, or restored, shape
stays."""
import os
import shutil
import subprocess

import numpy as np
import pytest

from nbodygo_gb300 import _abi as A
from nbodygo_gb300 import workloads as W
from nbodygo_gb300.api import Simulation

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
MIN_N = 98304


def test_rule(tmp_path):
    nvcc = shutil.which("nvcc") or ("/usr/local/cuda/bin/nvcc" if os.path.exists("/usr/local/cuda/bin/nvcc") else None)
    if nvcc is None:
        pytest.skip("nvcc not available")
    exe = str(tmp_path / "default_shape")
    cmd = [nvcc, "-std=c++17", "-O1", "-I", os.path.join(ROOT, "nbodygo_gb300", "csrc"), "-I",
           os.path.join(ROOT, "include"), os.path.join(ROOT, "tests", "cpp", "default_shape.cu"), "-o", exe]
    r = subprocess.run(cmd, capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    r = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0 and "default shape bad 0" in r.stdout, r.stdout + r.stderr


def run(b, shape=None, first=None):
    with Simulation("mixed", capacity=len(b["x"]) + 8, seed=4) as s:
        if shape is not None:
            s.set_option(A.OPT_MIX_SHAPE, shape)
        if first is not None:
            s.set_bodies(first)
            s.step(1e-5, 1.0, 1)
        s.set_bodies(b)
        s.step(1e-5, 1.0, 2)
        return s.state()


@pytest.mark.gpu
@pytest.mark.parametrize("n,shape", [(3000, 6), (32767, 6), (32768, 2), (MIN_N - 512, 2), (MIN_N, A.MIX_SYM)])
def test_default_is_the_rules_shape(n, shape):
    b = W.uniform_ball(n)
    small, large = W.uniform_ball(2000), W.uniform_ball(MIN_N + 5)
    ref = run(b, shape=shape)
    for first in (None, small, large):
        got = run(b, first=first)
        for f in ("x", "vx", "fy"):
            assert np.array_equal(got[f], ref[f]), f


@pytest.mark.gpu
def test_a_given_or_restored_shape_stays():
    b = W.uniform_ball(MIN_N)
    ref = run(b, shape=7)
    again = run(b, shape=7, first=W.uniform_ball(1000))
    with Simulation("mixed", seed=4) as s, Simulation("mixed", seed=4) as t:
        s.set_option(A.OPT_MIX_SHAPE, 7)
        s.set_bodies(b)
        t.set_bodies(W.uniform_ball(10))
        t.load_state(s.save_state())
        t.step(1e-5, 1.0, 2)
        restored = t.state()
    for got in (again, restored):
        for f in ("x", "vx", "fy"):
            assert np.array_equal(got[f], ref[f]), f
