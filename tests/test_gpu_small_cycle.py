"""Collections on both sides of the capacity (4,096) below which one block runs
the cycle's start, events, compaction and order: bit-identical to a context of
a larger capacity, which takes the multi-block kernels, and, in the plain
form, to the oracle."""
import numpy as np
import pytest

from nbodygo_gb300 import _abi as A
from nbodygo_gb300 import workloads as W
from nbodygo_gb300.api import Simulation
from oracle.oracle import OracleSim

from helpers import assert_states_identical
from test_gpu_plain_parity import dense_cluster

pytestmark = pytest.mark.gpu


def _run(b, form, capacity, cycles, adds=None):
    s = Simulation(form, capacity=capacity, seed=3)
    s.set_bodies(b)
    if adds is not None:
        s.add_bodies(adds)
    s.step(0.02, 0.9, cycles)
    out = s.state()
    s.close()
    return out


@pytest.mark.parametrize("form", ["fp64", "mixed"])
@pytest.mark.parametrize("n", [1, 2, 31, 33, 127, 129, 400, 1025])
def test_small_and_large_capacity_agree(n, form):
    """Fragments, merges, removals and adds every cycle; in the mixed form the
    order is sorted, carried and sorted again."""
    b = dense_cluster(n, seed=500 + n)
    adds = {k: v[: min(n, 3)].copy() for k, v in dense_cluster(max(n, 3), seed=900).items()}
    adds["id"] = np.arange(10 ** 6, 10 ** 6 + len(adds["x"]), dtype=np.int64)
    small = _run(b, form, 64, 6, adds)
    large = _run(b, form, 5000, 6, adds)
    for f in small:
        x, y = small[f], large[f]
        assert x.shape == y.shape and x.tobytes() == y.tobytes(), f


def test_small_cycle_matches_the_oracle():
    b = dense_cluster(300, seed=21)
    s = Simulation("fp64", capacity=64, seed=9)
    s.set_bodies(b)
    o = OracleSim(seed=9, threads=8)
    o.set_bodies(b)
    for _ in range(5):
        s.step(0.05, 0.9, 1)
        o.step(0.05, 0.9, 1)
        assert_states_identical(s.state(), o.state())
    s.close()


@pytest.mark.parametrize("n", [4095, 4096, 4097, 8193, 40961, 131073])
def test_order_of_every_sort(n):
    """Forces with the one-block, the fused and the multi-launch sort: within
    the form's bound of the plain form's, and the same on a second pass."""
    b = W.plummer(n, seed=33)
    b["collision"][:] = A.NONE
    with Simulation("mixed", capacity=n) as s:
        s.set_bodies(b)
        f = np.stack(s.force_pass())
        g = np.stack(s.force_pass())
    assert f.tobytes() == g.tobytes()
    k = np.arange(0, n, max(1, n // 40))
    x = np.stack([b["x"], b["y"], b["z"]])
    for i in k:
        d = x - x[:, i:i + 1]
        r = np.sqrt((d * d).sum(0))
        w = np.where(r > b["radius"] + b["radius"][i], b["mass"] / np.maximum(r, 1e-90) ** 3, 0.0)
        t = W.G * b["mass"][i] * w * d
        assert np.linalg.norm(f[:, i] - t.sum(1)) <= 1e-6 * np.linalg.norm(t, axis=0).sum()
