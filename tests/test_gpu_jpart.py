"""The symmetric kernel's j partials: asked for by the mixed direct sum alone,
whatever shape a context of another form has, and given back when the default
shape of a load is one-sided.  The failure hook stands in for a device without
room for them."""
import numpy as np
import pytest

from nbodygo_gb300 import _abi as A
from nbodygo_gb300 import workloads as W
from nbodygo_gb300.api import NbgError, Simulation

pytestmark = pytest.mark.gpu


def free_bytes():
    torch = pytest.importorskip("torch")
    return torch.cuda.mem_get_info(0)[0]


@pytest.mark.parametrize("n", [3000, 6000])
@pytest.mark.parametrize("prec,bh", [("fp64", 0), ("fp64", 1), ("mixed", 1), ("mixed", 0)])
def test_only_the_direct_sum_asks(prec, bh, n):
    with Simulation(prec, capacity=n) as s:
        s.set_option(A.OPT_BARNES_HUT, bh)
        s.set_option(A.OPT_MIX_SHAPE, A.MIX_SYM)
        s.set_option(A.OPT_TEST_FAIL_JPART, 1)
        s.set_bodies(W.plummer(n=n, seed=1))
        if prec == "mixed" and not bh:
            for call in (s.force_pass, lambda: s.step(1e-3, 1.0, 1)):
                with pytest.raises(NbgError):
                    call()
            s.set_option(A.OPT_TEST_FAIL_JPART, 0)
        s.force_pass()
        assert s.step(1e-3, 1.0, 2)["steps_done"] == 2


def test_an_octree_context_takes_no_memory_for_them():
    b = W.uniform_ball(200000)  # 76,636 block pairs: 589 MB with the quarter to spare
    with Simulation("mixed", capacity=200001) as s:
        s.set_option(A.OPT_BARNES_HUT, 1)
        s.set_bodies(b)
        before = free_bytes()
        s.step(1e-5, 1.0, 1)
        assert before - free_bytes() < 300 << 20


def test_a_one_sided_default_gives_them_back():
    with Simulation("mixed", capacity=98305) as s:
        s.set_bodies(W.uniform_ball(98304))  # 18,528 block pairs: 142 MB
        before = free_bytes()
        s.step(1e-5, 1.0, 1)
        held = before - free_bytes()
        assert held > 100 << 20
        s.set_bodies(W.uniform_ball(3000))
        assert before - free_bytes() < held - (100 << 20)
        s.step(1e-5, 1.0, 1)
        s.set_bodies(W.uniform_ball(98304))
        assert s.step(1e-5, 1.0, 2)["steps_done"] == 2


@pytest.mark.parametrize("n", [45000, 65536, 81920])
def test_autotune_passes_over_a_shape_without_room(n, tmp_path):
    """Sizes where the one-sided shape that would run in a symmetric one's
    place is among the fastest, so a time recorded under the wrong name is
    chosen in most of the tries."""
    for k in range(4):
        cache = str(tmp_path / f"cache{k}")
        with Simulation("mixed", capacity=n) as s:
            s.set_option(A.OPT_TEST_FAIL_JPART, 1)
            s.set_bodies(W.plummer(n=n, seed=1))
            shape = s.autotune(cache)[0]
            assert shape not in (A.MIX_SYM, A.MIX_SYM + 1)
            assert int(open(cache).read().split()[1]) == shape
            assert s.step(1e-5, 1.0, 2)["steps_done"] == 2


def test_a_restored_shape_is_kept_or_refused():
    """A resumed run continues bit for bit or not at all; a shape that the
    rule chose gives way."""
    b = W.uniform_ball(98304)
    with Simulation("mixed", seed=2) as s, Simulation("mixed") as t:
        s.set_bodies(b)
        s.step(1e-5, 1.0, 1)
        snap = s.save_state()
        s.step(1e-5, 1.0, 2)
        t.set_option(A.OPT_TEST_FAIL_JPART, 1)
        t.load_state(snap)
        for call in (t.force_pass, lambda: t.step(1e-5, 1.0, 2)):
            with pytest.raises(NbgError):
                call()
        t.load_state(snap)
        t.set_option(A.OPT_TEST_FAIL_JPART, 0)
        t.step(1e-5, 1.0, 2)
        want, got = s.state(), t.state()
        for f in ("x", "vx", "fy"):
            assert np.array_equal(got[f], want[f]), f
    with Simulation("mixed", seed=2) as s:
        s.set_option(A.OPT_TEST_FAIL_JPART, 1)
        s.set_bodies(b)
        assert s.step(1e-5, 1.0, 2)["steps_done"] == 2


def test_a_load_whose_shape_has_no_room_leaves_an_empty_context():
    """The default shape of the new collection needs larger partial sums: if
    they do not fit, the load fails and no old count stands beside new bodies."""
    small, large = W.uniform_ball(3000), W.uniform_ball(98304)
    with Simulation("mixed", capacity=98305, seed=6) as s, Simulation("mixed", capacity=98305, seed=6) as t:
        s.set_bodies(small)
        s.step(1e-5, 1.0, 1)
        s.set_option(A.OPT_TEST_FAIL_JPART, 2)
        with pytest.raises(NbgError):
            s.set_bodies(large)
        assert s.count() == 0 and len(s.state()["x"]) == 0
        s.set_option(A.OPT_TEST_FAIL_JPART, 0)
        assert s.step(1e-5, 1.0, 2)["n_bodies"] == 0
        for c in (s, t):
            c.set_bodies(large)
            c.step(1e-5, 1.0, 2)
        got, want = s.state(), t.state()
        for f in ("x", "vx", "fy"):
            assert np.array_equal(got[f], want[f]), f
