"""Every body's force, in every kernel shape of the mixed form, against the sum
of the magnitudes of its pair forces: a share of a body's sum that goes missing
in one chunk is far above this bound, and may be far below a relative L2 over
all bodies.  Counts that leave every segment of a chunk short."""
import numpy as np
import pytest

from nbodygo_gb300 import _abi as A
from nbodygo_gb300 import workloads as W
from nbodygo_gb300.api import Simulation

pytestmark = pytest.mark.gpu
# Bound on the error of an FP32 pair term, relative to the term.  A pair further
# than kappa = 0.05 of the offset from the tile's origin is off by at most
# 2^-24 (2 / kappa + 1) of its distance in each coordinate, 4.3e-6 in all, which
# counts twice, and 3 x 2^-22 for the reciprocal root and the products.
TERM = 1e-5


def magnitudes(b):
    x = np.stack([b[c] for c in "xyz"])
    out = np.zeros(x.shape[1])
    for i0 in range(0, len(out), 256):
        d = x[:, None, :] - x[:, i0:i0 + 256, None]
        r2 = (d * d).sum(0)
        r2[r2 == 0] = np.inf
        out[i0:i0 + 256] = (b["mass"] / r2).sum(1)
    return W.G * b["mass"] * out


@pytest.mark.parametrize("kind", ["plummer", "ball"])
@pytest.mark.parametrize("n", [33, 257, 513, 700, 1000, 2501])
def test_every_body_in_every_shape(n, kind):
    b = W.plummer(n=n, seed=n) if kind == "plummer" else W.uniform_ball(n, seed=n)
    with Simulation("fp64") as s:
        s.set_bodies(b)
        g = np.array(s.force_pass())
    scale = magnitudes(b)
    with Simulation("mixed") as s:
        for shape in range(A.MIX_SHAPES):
            s.set_option(A.OPT_MIX_SHAPE, shape)
            s.set_bodies(b)
            err = np.sqrt(((np.array(s.force_pass()) - g) ** 2).sum(0)) / scale
            assert err.max() <= TERM, (shape, int((err > TERM).sum()), float(err.max()))
