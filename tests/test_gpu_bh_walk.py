"""The mixed Barnes-Hut walk at the edges of its groups, lists and stack,
against the FP64 tree on the same bodies (the bound of the form's other
tests: relative L2 1e-5, median 1e-6 per body)."""
import numpy as np
import pytest

from nbodygo_gb300 import _abi as A
from nbodygo_gb300 import workloads as W
from nbodygo_gb300.api import Simulation
from oracle.oracle import OracleSim

pytestmark = pytest.mark.gpu


def _forces(b, form, shape=0):
    with Simulation(form) as s:
        s.set_option(A.OPT_BARNES_HUT, 1)
        s.set_option(A.OPT_BH_SHAPE, shape)
        s.set_bodies(b)
        f = np.stack(s.force_pass())
        terms = s.step(0.0, 1.0, 1)["bh_terms"]
    return f, terms


def _close(b, shape=0):
    g, tg = _forces(b, "fp64")
    f, tf = _forces(b, "mixed", shape)
    mag = np.linalg.norm(g, axis=0)
    err = np.linalg.norm(f - g, axis=0)
    assert np.linalg.norm(f - g) <= 1e-5 * np.linalg.norm(g)
    if len(mag) > 2:
        assert np.median(err[mag > 0] / mag[mag > 0]) <= 1e-6
    # a body's opening tests differ from the FP64 ones only at ties
    assert abs(tf - tg) <= 1e-4 * tg + 8


def _clustered(n, seed):
    """Half the bodies in cells far below the tree's 2^-20 resolution: leaves
    that hold several bodies, long thin descents."""
    b = W.plummer(n, seed=seed)
    r = W.SplitMix64(seed + 9)
    for c in ("x", "y", "z"):
        h = n // 2
        b[c][h:] = b[c][: n - h][np.arange(n - h) // 5] + r.uniform(n - h, 1e-5, 2e-4)
    b["collision"][:] = A.NONE
    b["radius"][:] = 0.0
    return b


@pytest.mark.parametrize("shape", [0, 1, 2])
@pytest.mark.parametrize("n", [1, 2, 31, 32, 33, 127, 129, 1000, 5003])
def test_small_collections(n, shape):
    b = W.plummer(n, seed=50 + n)
    b["collision"][:] = A.NONE
    _close(b, shape)


@pytest.mark.parametrize("n", [59999, 60000, 60033])
def test_both_sides_of_a_warp_to_a_group(n):
    b = W.plummer(n, seed=6)
    b["collision"][:] = A.NONE
    _close(b)


@pytest.mark.parametrize("n", [64, 3000, 70001])
def test_shared_leaves(n):
    _close(_clustered(n, 70 + n))


@pytest.mark.parametrize("scale,mass", [(1e60, 1e70), (1e-30, 1e-10), (1.0, 1e-90), (1e25, 1.0)])
def test_fp64_walk_out_of_fp32_range(scale, mass):
    """Coordinates and masses that FP32 cannot hold: the bodies decide in
    FP64, and terms outside nbg_exact.h's range take the ordinary operators."""
    b = W.plummer(700, seed=12)
    for c in "xyz":
        b[c] *= scale
    b["mass"][:] = mass
    b["radius"][:] = 0.0
    b["collision"][:] = A.NONE
    f, _ = _forces(b, "fp64")
    o = OracleSim(threads=8)
    o.set_barnes_hut(True)
    o.set_bodies(b)
    g = np.stack(o.forces())
    mag, err = np.linalg.norm(g / np.abs(g).max(), axis=0), np.linalg.norm((f - g) / np.abs(g).max(), axis=0)
    assert np.all(err <= 1e-12 * mag)


@pytest.mark.parametrize("n", [1, 2, 31, 32, 33, 65, 500, 4001])
def test_fp64_walk_matches_the_oracle(n):
    b = W.plummer(n, seed=80 + n)
    b["collision"][:] = A.NONE
    f, _ = _forces(b, "fp64")
    o = OracleSim(threads=8)
    o.set_barnes_hut(True)
    o.set_bodies(b)
    g = np.stack(o.forces())
    assert np.all(np.linalg.norm(f - g, axis=0) <= 1e-12 * np.linalg.norm(g, axis=0))
