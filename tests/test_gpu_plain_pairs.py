"""The plain form's pair pass at the edges of its blocks and tiles and with
operands its straight path hands to the ordinary operators, bit for bit
against the oracle."""
import numpy as np
import pytest

from nbodygo_gb300 import _abi as A
from nbodygo_gb300 import workloads as W
from nbodygo_gb300.api import Simulation
from oracle.oracle import OracleSim

from test_gpu_plain_parity import dense_cluster

pytestmark = pytest.mark.gpu


def _bits(a):
    return np.ascontiguousarray(a, dtype=np.float64).view(np.uint64)


def _same_forces(b):
    with Simulation("fp64") as s:
        s.set_bodies(b)
        f = s.force_pass()
    o = OracleSim(threads=8)
    o.set_bodies(b)
    for got, exp in zip(f, o.forces()):
        nan = np.isnan(exp)
        assert np.array_equal(nan, np.isnan(got))
        assert np.array_equal(_bits(got)[~nan], _bits(exp)[~nan])


@pytest.mark.parametrize("n", [1, 2, 3, 4, 5, 31, 32, 33, 191, 192, 193, 385, 1215, 1217, 2433, 9729])
def test_block_and_tile_edges(n):
    _same_forces(W.plummer(n, seed=200 + n))


@pytest.mark.parametrize("kind", ["planar", "lattice", "coincident", "massless", "negative", "tiny", "huge", "mixed"])
def test_operands(kind):
    n = 400
    b = W.plummer(n, seed=9)
    r = W.SplitMix64(77)
    if kind == "planar":
        b["z"][:] = 0.0
    elif kind == "lattice":  # differences, squares and roots with few bits: ties
        for c in "xyz":
            b[c][:] = np.floor(r.uniform(n, -40, 40)) * 0.25
        b["mass"][:] = 2.0 ** np.floor(r.uniform(n, 0, 30))
        b["radius"][:] = 0.0
    elif kind == "coincident":
        for c in "xyz":
            b[c][n // 2:] = b[c][: n - n // 2]
    elif kind == "massless":
        b["mass"][::3] = 0.0
    elif kind == "negative":
        b["mass"][::3] *= -1.0
        b["radius"][::5] = -1.0
    elif kind == "tiny":
        for c in "xyz":
            b[c] *= 1e-60
        b["mass"][:] *= 1e-80
        b["radius"][:] = 1e-65
    elif kind == "huge":
        for c in "xyz":
            b[c] *= 1e60
        b["mass"][:] = 1e70
        b["x"][::7] = 1e300
    else:
        b["x"][3] = np.nan
        b["y"][5] = np.inf
        b["radius"][9] = np.nan
        b["radius"][11] = np.inf
        b["mass"][13] = 1e-310
        b["x"][15] = b["x"][16] + 5e-320
    _same_forces(b)


def test_collections_of_every_size_bit_exact():
    """Blocks are cut within collections: sizes around a block and a tile."""
    sizes = [1, 0, 3, 4, 5, 63, 64, 65, 191, 193, 700, 2, 1500]
    sims = [{f: v[:n] for f, v in dense_cluster(max(n, 1), seed=300 + k).items()} for k, n in enumerate(sizes)]
    with Simulation("fp64", seed=11) as s:
        s.set_collections(sims)
        s.step(0.01, 0.9, 2)
        got, counts = s.state(), s.sim_counts()
    o = 0
    for k, (b, c) in enumerate(zip(sims, counts)):
        if len(b["x"]) == 0:
            assert c == 0
            continue
        ora = OracleSim(seed=11, threads=8)
        ora.set_bodies(b)
        ora.step(0.01, 0.9, 2)
        e = ora.state()
        m = len(e["x"])
        assert m == c
        for f in ("x", "y", "z", "vx", "vy", "vz", "mass"):
            assert np.array_equal(_bits(got[f][o:o + m]), _bits(e[f])), (k, f)
        o += m
