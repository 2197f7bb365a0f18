"""Radii so large that every pair of a collection is near, in the mixed form:
an infinite one, and ones whose near-pair distance is past the far-away places
that fill up a short tile.  Odd counts leave every tile short; the events must
be the plain form's, the forces within the mixed tolerance, and no body may meet
one of the next collection."""
import numpy as np
import pytest

from nbodygo_gb300 import _abi as A
from nbodygo_gb300 import workloads as W
from nbodygo_gb300.api import Simulation

from helpers import assert_events_identical, rel_l2

pytestmark = pytest.mark.gpu
TOL = 1e-6  # relative L2, as for the mixed form elsewhere


def with_radii(n, seed, radii, behavior):
    b = W.plummer(n=n, seed=seed, behavior=behavior)
    for k, r in enumerate(radii):
        b["radius"][(n // 2 + 3 * k) % n] = r
    return b


def forces_and_events(prec, sims, shape, capacity):
    with Simulation(prec, capacity=capacity, seed=3) as s:
        if shape is not None and prec == "mixed":
            s.set_option(A.OPT_MIX_SHAPE, shape)
        s.set_collections(sims)
        f = np.array(s.force_pass())
        s.step(1e-3, 0.9, 1)
        return f, s.events()


@pytest.mark.parametrize("radii", [(np.inf,), (1e19,), (2e18, 3e18), (np.inf, 1e19)])
@pytest.mark.parametrize("shape", [None, 0, 2, 7, 12, 17, A.MIX_SYM])
def test_near_everything(radii, shape):
    for behavior in (A.SUBSUME, A.ELASTIC):
        sims = [with_radii(5, 1, radii, behavior), W.plummer(n=7, seed=2, behavior=behavior),
                with_radii(301, 3, radii, behavior), W.plummer(n=131, seed=4, behavior=behavior)]
        f, ev = forces_and_events("mixed", sims, shape, 0)
        g, want = forces_and_events("fp64", sims, None, 0)
        assert len(want) > 0
        assert_events_identical(ev, want)
        o = 0
        for b in sims:
            n = len(b["x"])
            assert rel_l2(f[:, o:o + n], g[:, o:o + n]) <= TOL
            o += n


@pytest.mark.parametrize("shape", [2, A.MIX_SYM])
def test_near_everything_with_thresholds_by_tile(shape):
    sims = [with_radii(3001, 5, (np.inf,), A.SUBSUME)]
    f, ev = forces_and_events("mixed", sims, shape, 40000)
    g, want = forces_and_events("fp64", sims, None, 0)
    assert len(want) > 0
    assert_events_identical(ev, want)
    assert rel_l2(f, g) <= TOL
