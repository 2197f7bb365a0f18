"""Near-pair thresholds by tile (k_mix_reach, from 32,768 bodies on; the
symmetric kernel's per pair of blocks): a disk around a large body, with other
large bodies among the small ones and overlaps of every kind of pair.  The
events must be the plain form's, the forces within the mixed tolerance, with
and without the per-tile thresholds."""
import numpy as np
import pytest

from nbodygo_gb300 import _abi as A
from nbodygo_gb300 import workloads as W
from nbodygo_gb300.api import Simulation

from helpers import assert_events_identical, rel_l2

pytestmark = pytest.mark.gpu
TOL = 1e-6


def crowded_disk(n):
    b = W.disk(n=n, seed=17)
    rng = W.SplitMix64(91)
    big = np.arange(5, n, n // 7)                     # large bodies among the small
    b["radius"][big] = rng.uniform(len(big), 6.0, 40.0)
    k = np.arange(11, n, n // 60)                     # bodies at the edge of a large one: just in, just out
    host = big[np.arange(len(k)) % len(big)]
    d = (b["radius"][host] + b["radius"][k]) * (1.0 + np.where(np.arange(len(k)) % 2, 1e-9, -1e-9))
    for c, u in zip("xyz", (0.6, 0.0, 0.8)):
        b[c][k] = b[c][host] + u * d
    j = np.arange(23, n, n // 90)                     # overlapping small neighbours
    b["x"][j] = b["x"][j - 1] + 0.5
    b["y"][j], b["z"][j] = b["y"][j - 1], b["z"][j - 1]
    return b


@pytest.mark.parametrize("n,cap", [(32767, 32767), (32768, 32768), (20001, 40000)])
@pytest.mark.parametrize("shape", [0, 2, A.MIX_SYM])
def test_large_bodies_among_small(n, cap, shape):
    b = crowded_disk(n)
    out = []
    for prec in ("fp64", "mixed"):
        with Simulation(prec, capacity=cap, seed=3) as s:
            if prec == "mixed":
                s.set_option(A.OPT_MIX_SHAPE, shape)
            s.set_bodies(b)
            f = np.array(s.force_pass())
            s.step(0.001, 0.9, 1)
            out.append((f, s.events()))
    assert len(out[0][1]) > 60
    assert_events_identical(out[1][1], out[0][1])
    assert rel_l2(out[1][0][:, 1:], out[0][0][:, 1:]) <= TOL
