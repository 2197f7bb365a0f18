"""The heaviest body of a collection of at most 4,096: the one-sided mixed
kernels leave its pull to the last kernel, which adds it in FP64.  Around a
star, what is left of a body's error is that of its neighbours' FP32 terms, so
it is held against their magnitudes and not against the star's pull; the
overlaps and events are the plain form's."""
import numpy as np
import pytest

from nbodygo_gb300 import _abi as A
from nbodygo_gb300 import workloads as W
from nbodygo_gb300.api import Simulation

from helpers import assert_events_identical

pytestmark = pytest.mark.gpu
LIMIT = 4096
# Bound on the error of a neighbour's FP32 term, relative to the term.  A pair
# further than kappa = 0.05 of the offset from the tile's origin is off by at most
# 2^-24 (2 / kappa + 1) of its distance in each coordinate, 4.3e-6 in all, which
# counts twice, and 3 x 2^-22 for the reciprocal root and the products.
TERM = 1e-5


def forces(prec, sims, shape=None, step=True):
    with Simulation(prec, seed=3) as s:
        if shape is not None and prec == "mixed":
            s.set_option(A.OPT_MIX_SHAPE, shape)
        s.set_collections(sims)
        f = np.array(s.force_pass())
        if step:
            s.step(1e-3, 0.9, 1)
        return f, s.events()


def magnitudes(b, skip=None):
    """Each body's sum of pair force magnitudes, body `skip` left out as a source."""
    x = np.stack([b[c] for c in "xyz"])
    m = b["mass"].copy()
    if skip is not None:
        m[skip] = 0.0
    out = np.zeros(x.shape[1])
    for i0 in range(0, len(out), 512):
        d = x[:, None, :] - x[:, i0:i0 + 512, None]
        r2 = (d * d).sum(0)
        r2[r2 == 0] = np.inf
        out[i0:i0 + 512] = (m / r2).sum(1)
    return W.G * b["mass"] * out


def check(b, f, g, star):
    err = np.sqrt(((f - g) ** 2).sum(0))
    pull = np.sqrt((g ** 2).sum(0))
    bound = TERM * magnitudes(b, star) + 2.0 ** -40 * pull
    bound[star] = TERM * magnitudes(b)[star]
    assert np.all(err <= bound), (err / bound).max()


@pytest.mark.parametrize("n", [2, 31, 300, 513, 1000, 2049, LIMIT])
@pytest.mark.parametrize("shape", [None, 0, 7, 12, 17])
def test_disk_around_a_star(n, shape):
    b = W.disk(n=n, seed=n)
    star = int(np.argmax(b["mass"]))
    k = np.arange(n)[np.arange(n) != star][::9]
    b["x"][k[:3]], b["y"][k[:3]], b["z"][k[:3]] = b["x"][star] + 5.0, b["y"][star], b["z"][star]  # inside it
    f, ev = forces("mixed", [b], shape)
    g, want = forces("fp64", [b])
    assert_events_identical(ev, want)
    check(b, f, g, star)


def test_several_collections_and_sizes_past_the_limit():
    """The heaviest body of each; past the limit the pair kernel's own terms."""
    sims = [W.disk(n=700, seed=1), W.disk(n=LIMIT + 1, seed=2), W.plummer(n=33, seed=3), W.disk(n=LIMIT, seed=4)]
    sims[0]["mass"] *= 1e-20  # below FP32's range beside the others' stars
    f, ev = forces("mixed", sims)
    g, want = forces("fp64", sims)
    assert_events_identical(ev, want)
    o = 0
    for k, b in enumerate(sims):
        n = len(b["x"])
        star = int(np.argmax(b["mass"]))
        if k < 2:
            assert np.sqrt(((f - g)[:, o:o + n] ** 2).sum() / (g[:, o:o + n] ** 2).sum()) <= 1e-6
        else:
            check(b, f[:, o:o + n], g[:, o:o + n], star)
        o += n


@pytest.mark.parametrize("what", ["fragmenting", "absent", "not finite", "none live"])
def test_no_pull_from_a_body_that_exerts_none(what):
    """The heaviest body is the heaviest that exists, is not fragmenting and
    has a finite position."""
    b = W.disk(n=500, seed=5)
    star = int(np.argmax(b["mass"]))
    if what == "fragmenting":
        b["flags"][star] |= A.F_FRAGMENTING
    elif what == "absent":
        b["flags"][star] = 0
    elif what == "not finite":
        b["x"][star] = np.nan
    else:
        b["flags"][:] |= A.F_FRAGMENTING
    live = (b["flags"] & (A.F_EXISTS | A.F_FRAGMENTING)) == A.F_EXISTS
    live[star] &= what != "not finite"
    f, _ = forces("mixed", [b], step=False)
    g, _ = forces("fp64", [b], step=False)
    b["mass"][~live] = 0.0
    b["x"][~live] = 0.0  # of the sums below
    err = np.sqrt(((f - g) ** 2).sum(0))
    assert np.all(err[live] <= (TERM * magnitudes(b, star))[live] + 2.0 ** -40 * np.sqrt((g ** 2).sum(0))[live])
