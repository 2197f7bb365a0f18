"""The ends of the near-pair thresholds' range, formed in FP32 against the other
block's (k_pair_sym) or the tiles' in reach (k_mix_reach) largest radius."""
import numpy as np
import pytest

from nbodygo_gb300 import _abi as A
from nbodygo_gb300 import workloads as W
from nbodygo_gb300.api import Simulation

from helpers import assert_events_identical, rel_l2
from test_gpu_near_reach import crowded_disk

pytestmark = pytest.mark.gpu


def run(prec, b, shape, capacity=0, sims=None):
    with Simulation(prec, capacity=capacity, seed=3) as s:
        if prec == "mixed":
            s.set_option(A.OPT_MIX_SHAPE, shape)
        s.set_collections([b] + (sims or []))
        f = np.array(s.force_pass())[:, :len(b["x"])]
        s.step(0.0, 1.0, 1)
        return f, s.events()


@pytest.mark.parametrize("n,shape,capacity", [(513, A.MIX_SYM, 0), (1025, A.MIX_SYM + 1, 0), (257, 2, 40000),
                                              (513, 0, 40000)])
def test_a_tiny_system_of_points(n, shape, capacity):
    """A ball of radius 1e-10 without radii whose last tile is one body on its
    own origin, at a position that FP32 holds exactly (no low part).  Beside
    it, for the one-sided shapes, a collection with a larger radius."""
    b = W.uniform_ball(n, seed=7, R=1e-10, radius=0.0)
    for c in "xyz":
        b[c][:] = b[c].astype(np.float32)
    other = W.uniform_ball(n, seed=8, R=1e-10, radius=1e-20)
    sims = [other] if capacity else None
    f, _ = run("mixed", b, shape, capacity, sims)
    g, _ = run("fp64", b, shape, 0, sims)
    assert np.all(np.isfinite(f)) and rel_l2(f, g) <= 1e-6


@pytest.mark.parametrize("shape", [0, 2, A.MIX_SYM, A.MIX_SYM + 1])
@pytest.mark.parametrize("gap", [1.75e19, 1.8e19])
def test_blocks_at_the_end_of_fp32s_range(shape, gap):
    """Two blocks so far apart that the squared distance is just below FP32's
    largest value, and two bodies whose radii reach from one to the other."""
    b = W.uniform_ball(1024, seed=9, R=1e6, radius=1.0, behavior=A.ELASTIC)
    b["x"][512:] += gap
    b["radius"][100], b["radius"][700] = 1.0e19, 0.95e19
    _, ev = run("mixed", b, shape)
    _, want = run("fp64", b, shape)
    assert len(want) > 0
    assert_events_identical(ev, want)


@pytest.mark.parametrize("shape", [0, 2])
def test_large_bodies_without_thresholds_by_tile(shape):
    """A capacity below the one from which k_mix_reach runs: every threshold
    is against the largest radius of all."""
    b = crowded_disk(16001)
    f, ev = run("mixed", b, shape, 16384)
    g, want = run("fp64", b, shape, 16384)
    assert len(want) > 60
    assert_events_identical(ev, want)
    assert rel_l2(f[:, 1:], g[:, 1:]) <= 1e-6
