"""The Barnes-Hut build's sort, in its two forms and at its tiles' edges, bit for
bit against each other."""
import numpy as np
import pytest

from nbodygo_gb300 import _abi as A
from nbodygo_gb300 import workloads as W
from nbodygo_gb300.api import Simulation

pytestmark = pytest.mark.gpu


def bh_forces(cap, sims):
    with Simulation("fp64", capacity=cap) as s:
        s.set_option(A.OPT_BARNES_HUT, 1)
        s.set_collections(sims)
        return np.array(s.force_pass())


@pytest.mark.parametrize("sizes", [[1], [1023], [1024], [1025], [5000], [700, 1, 324, 2100]])
def test_both_forms_of_the_sort(sizes):
    sims = [W.plummer(n, seed=n + k) if n > 1 else W.uniform_ball(n) for k, n in enumerate(sizes)]
    narrow, wide = bh_forces(sum(sizes), sims), bh_forces(400000, sims)
    assert np.array_equal(narrow, wide, equal_nan=True)


def test_a_full_wide_sort_matches_the_oracle_on_a_part():
    """260,000 bodies, of which most are far away in a second collection: the
    first collection's forces are those it has alone."""
    small, large = W.plummer(3001, seed=2), W.uniform_ball(257000, R=900.0)
    both = bh_forces(260001, [small, large])
    assert np.array_equal(both[:, :3001], bh_forces(3001, [small]))
