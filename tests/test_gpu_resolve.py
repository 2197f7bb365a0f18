"""Collision resolution by warps: pairs that collide head on, grazing, with an
axis-aligned or zero approach, with fragmenting and massless partners, alone,
a few at once (a warp to each), around the switch to a thread to each and in
chains through one body, bit for bit as the oracle resolves them."""
import numpy as np
import pytest

from nbodygo_gb300 import _abi as A
from nbodygo_gb300 import workloads as W
from nbodygo_gb300.api import Simulation
from oracle.oracle import OracleSim

from helpers import assert_events_identical, assert_states_identical, body_set

pytestmark = pytest.mark.gpu


def touching_pairs(k, seed, chain=False):
    """k overlapping pairs far from each other, or a row of k + 1 bodies each
    overlapping the next."""
    rng = W.SplitMix64(seed)
    n = k + 1 if chain else 2 * k
    b = body_set([{}] * n)
    u = rng.uniform(6 * n, -1.0, 1.0).reshape(6, n)
    for q in range(n):
        pair = q // 2
        if chain:
            b["x"][q] = 1.7 * q
        else:
            b["x"][q] = 1000.0 * pair + (q % 2) * (1.0 + 0.4 * u[0, q])
            kind = pair % 5
            if q % 2 and kind != 1:                       # kind 1: separated along x alone
                b["y"][q], b["z"][q] = 0.5 * u[1, q], 0.5 * u[2, q]
            if q % 2 and kind == 2:                       # along z alone
                b["x"][q], b["y"][q], b["z"][q] = 1000.0 * pair, 0.0, 1.3
    b["vx"][:], b["vy"][:], b["vz"][:] = 5 * u[3], 5 * u[4], 5 * u[5]
    if not chain:
        still = np.arange(6, n - 1, 10)                   # equal velocities: no relative speed
        for c in ("vx", "vy", "vz"):
            b[c][still + 1] = b[c][still]
        along = np.arange(8, n - 1, 10)                   # relative velocity along x alone
        b["vy"][along + 1], b["vz"][along + 1] = b["vy"][along], b["vz"][along]
    b["mass"][:] = rng.log_uniform(n, 1e3, 1e9)
    b["mass"][n // 3::11] = 0.0
    b["radius"][:] = 1.0
    beh = np.array([A.ELASTIC, A.ELASTIC, A.FRAGMENT, A.ELASTIC, A.SUBSUME], dtype=np.int32)
    b["collision"][:] = beh[np.floor(rng.uniform(n, 0, 5)).astype(int)]
    b["frag_factor"][:] = rng.uniform(n, 0.0, 1.0)
    b["frag_step"][:] = rng.uniform(n, 0.0, 4.0)
    return b


@pytest.mark.parametrize("k,chain", [(1, False), (2, False), (3, False), (8, False), (9, False), (60, False),
                                     (200, False), (1, True), (2, True), (9, True), (300, True)])
@pytest.mark.parametrize("seed", [1, 2])
def test_resolution_is_the_oracles(k, chain, seed):
    b = touching_pairs(k, 100 * seed + k, chain)
    with Simulation("fp64", seed=7) as s:
        s.set_bodies(b)
        o = OracleSim(seed=7, threads=4)
        o.set_bodies(b)
        for c in range(3):
            s.step(0.01, 0.8, 1)
            o.step(0.01, 0.8, 1)
            assert_events_identical(s.events(), o.events(), f"cycle {c}")
            assert_states_identical(s.state(), o.state(), where=f"cycle {c}")
