"""The plain pair pass over several collections: blocks of 4 to 32 bodies and
tiles of whole rounds, as the batch's total decides, at sizes around a round, a
64-body tile and a j tile.  Forces are the oracle's for each collection alone,
bit for bit."""
import numpy as np
import pytest

from nbodygo_gb300 import workloads as W
from nbodygo_gb300.api import Simulation
from oracle.oracle import OracleSim

pytestmark = pytest.mark.gpu
SIZES = (1, 7, 8, 9, 31, 33, 47, 48, 49, 63, 64, 65, 95, 97, 129, 191, 192, 193, 385)


@pytest.mark.parametrize("copies", [1, 6, 24, 96])
def test_every_size_in_every_cut(copies):
    sims = [W.plummer(n, seed=100 + n) for n in SIZES]
    want = []
    for b in sims:
        o = OracleSim(threads=8)
        o.set_bodies(b)
        want.append(np.array(o.forces()))
    with Simulation("fp64") as s:
        s.set_collections(sims * copies)
        f = np.array(s.force_pass())
    o = 0
    for k in range(copies):
        for n, w in zip(SIZES, want):
            assert np.array_equal(f[:, o:o + n].view(np.uint64), w.view(np.uint64)), (copies, k, n)
            o += n
