"""The mixed Barnes-Hut walk at the edges of its groups, lists and stack,
against the FP64 tree on the same bodies (the bound of the form's other
tests: relative L2 1e-5, median 1e-6 per body)."""
import numpy as np
import pytest

from nbodygo_gb300 import _abi as A
from nbodygo_gb300 import workloads as W
from nbodygo_gb300.api import Simulation

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
