"""Mixed form at the edges of its work cut: collections of less than a tile, a
tile and its neighbours, short last j tiles, and dense ones in which most
bodies take the careful pass, against the FP64 oracle."""
import numpy as np
import pytest

from nbodygo_gb300 import _abi as A
from nbodygo_gb300 import workloads as W
from nbodygo_gb300.api import Simulation
from oracle.oracle import OracleSim

from helpers import rel_l2
from test_gpu_plain_parity import dense_cluster

pytestmark = pytest.mark.gpu
# every term is rounded to 2^-24 of itself a few times and the sums are
# compensated: the form's stated bound, relative L2 1e-6
TOL = 1e-6


def _oracle(b, seed=5):
    o = OracleSim(seed=seed, threads=8)
    o.set_bodies(b)
    return o


@pytest.mark.parametrize("shape", [0, 2, 7, 12, 17])
@pytest.mark.parametrize("n", [1, 2, 33, 255, 256, 257, 511, 513, 1025, 2047, 4099])
def test_forces_at_tile_edges(n, shape):
    b = W.plummer(n=n, seed=100 + n)
    with Simulation("mixed") as s:
        s.set_option(A.OPT_MIX_SHAPE, shape)
        s.set_bodies(b)
        f = s.force_pass()
    g = _oracle(b).forces()
    if n == 1:
        assert all(np.all(c == 0) for c in f)
    else:
        assert rel_l2(f, g) <= TOL


@pytest.mark.parametrize("shape", [2, 7])
@pytest.mark.parametrize("n", [300, 700, 1500])
def test_careful_pass_events_exact(n, shape):
    """Most bodies of a dense cluster overlap others: forces within the bound
    and the first cycle's event list equal to the oracle's."""
    b = dense_cluster(n, seed=40 + n)
    with Simulation("mixed", seed=5) as s:
        s.set_option(A.OPT_MIX_SHAPE, shape)
        s.set_bodies(b)
        s.step(0.0, 0.9, 1)
        ev = s.events()
    o = _oracle(b)
    o.step(0.0, 0.9, 1)
    ref = o.events()
    assert len(ref) > 10
    for f in ("id1", "id2", "type"):
        assert np.array_equal(ev[f], ref[f])
