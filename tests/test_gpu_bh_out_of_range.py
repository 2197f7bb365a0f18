"""The mixed octree walk with bodies it cannot place in FP32: past its range,
with an infinite or NaN mass, or with moments that overflow.  The walk must
end.  A body at no FP32 distance makes every force NaN, as a leaf's term is;
where only a node's moment overflows, the node is opened for every body and
the forces on the light bodies are the direct sum's."""
import numpy as np
import pytest

from nbodygo_gb300 import _abi as A
from nbodygo_gb300 import workloads as W
from nbodygo_gb300.api import Simulation

from helpers import body_set, rel_l2

pytestmark = pytest.mark.gpu


def mixed_tree_forces(sims):
    with Simulation("mixed") as s:
        s.set_option(A.OPT_BARNES_HUT, 1)
        s.set_collections(sims)
        return np.array(s.force_pass())


@pytest.mark.parametrize("n", [2, 33, 1501])
@pytest.mark.parametrize("field,value", [("x", 1e39), ("z", -1e300), ("mass", np.inf), ("mass", np.nan)])
def test_the_walk_ends_and_every_force_is_nan(n, field, value):
    """Beside it, a collection in range keeps the forces it has alone."""
    b, other = W.plummer(n=n, seed=n), W.plummer(n=700, seed=5)
    b[field][n // 2] = value
    f = mixed_tree_forces([b, other])
    assert np.all(np.isnan(f[:, :n]).any(axis=0))
    assert np.array_equal(f[:, n:], mixed_tree_forces([other]))


@pytest.mark.parametrize("light", [20, 500])
def test_a_nodes_moment_overflows(light):
    """Two heavy bodies' moments overflow together, none alone, so every node
    with two of them is opened; the light ones' own masses vanish beside
    them.  What is left of the tree's error is FP32's."""
    rng = W.SplitMix64(3)
    n = 10 + light
    b = body_set([dict(radius=1.0) for _ in range(n)], behavior=A.NONE)
    for c in "xyz":
        b[c][:] = 1.2e10 + rng.uniform(n, -1e9, 1e9)
    b["mass"][:] = 1e-290
    b["mass"][:10] = 1e298
    f = mixed_tree_forces([b])[:, 10:]
    with Simulation("fp64") as s:
        s.set_bodies(b)
        g = np.array(s.force_pass())[:, 10:]
    assert np.all(np.isfinite(g)) and rel_l2(f, g) <= 1e-6
