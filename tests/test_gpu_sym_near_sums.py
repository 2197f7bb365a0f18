"""The symmetric kernel's exact sums over near pairs: a body's terms from one
block are added in FP64 and rounded once, on both sides of a unit.

Two shells of 512 bodies, a block each, so that every body lies well off its
tile's origin, and a near-pair factor that makes every pair a near one.  What
is left of the error is then the FP32 slot of the column side: half a unit in
the last place (2^-24) of the other shell's pull."""
import numpy as np
import pytest

from nbodygo_gb300 import _abi as A
from nbodygo_gb300 import workloads as W
from nbodygo_gb300.api import Simulation

from helpers import body_set

pytestmark = pytest.mark.gpu
B = 512


def shells(n, seed):
    rng = W.SplitMix64(seed)
    b = body_set([dict(radius=0.0) for _ in range(n)], behavior=A.NONE)
    for c, x in zip("xyz", rng.unit_vectors(n)):
        b[c][:] = x
    b["x"] += np.where(np.arange(n) < B, -1.25, 1.25)
    b["mass"][:] = 10.0 ** rng.uniform(n, 0.0, 6.0)
    return b


def pull(b, i, j):
    """Forces on the bodies i from the bodies j, in 64 bits and more."""
    x = np.stack([b[c] for c in "xyz"]).astype(np.longdouble)
    m = b["mass"].astype(np.longdouble)
    d = x[:, None, j] - x[:, i, None]
    r2 = (d * d).sum(0)
    w = np.where(r2 > 0, m[j] / np.where(r2 > 0, r2, 1) ** np.longdouble(1.5), 0)
    return W.G * m[i] * (w * d).sum(2)


@pytest.mark.parametrize("shape", [A.MIX_SYM, A.MIX_SYM + 1])
@pytest.mark.parametrize("seed,n", [(1, 2 * B), (2, 2 * B), (3, 2 * B - 31)])
def test_one_rounding_a_unit(shape, seed, n):
    b = shells(n, seed)
    with Simulation("mixed") as s:
        s.set_option(A.OPT_MIX_SHAPE, shape)
        s.set_option(A.OPT_NEAR_PPM, 10000000)
        s.set_bodies(b)
        f = np.array(s.force_pass())
    left, right = np.arange(B), np.arange(B, n)
    for own, other in ((left, right), (right, left)):
        cross, inside = pull(b, own, other), pull(b, own, own)
        scale = np.abs(cross).sum(0) + np.abs(inside).sum(0)
        err = np.abs(f[:, own] - (cross + inside))
        assert np.all(err <= 2.0 ** -24 * np.abs(cross) + 1e-11 * scale)
