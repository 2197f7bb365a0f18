"""The calls this framework is timed on.

A case is one call sequence of a program that steps collections held on the
host: load the bodies (set_bodies / set_collections_flat, from pinned arrays),
run some cycles (step) or one force pass (force_pass), read the state back.
The context, its form and options, and the pinned arrays are kept from call
to call, as such a program keeps them.

Bodies come from nbodygo_gb300.workloads, seeded.  A mixed-form case returns
what the next frame needs (ids, positions, velocities, masses, radii, flags);
a plain FP64 case, whose contract is bit parity, the forces too; the force
pass of the mixed form returns its forces in the 32 bits they are formed in.
"""
import math

import numpy as np
import torch

from nbodygo_gb300 import _abi as A
from nbodygo_gb300 import workloads
from nbodygo_gb300.api import Simulation

G = workloads.G
BEHAVIOR = {"none": A.NONE, "elastic": A.ELASTIC, "subsume": A.SUBSUME}
STATE = ("id", "x", "y", "z", "vx", "vy", "vz", "mass", "radius", "flags")
FORCES = ("fx", "fy", "fz")


def listed():
    return [
        # one interactive simulation in the reference's own arithmetic: the disk
        # around a central body, a second of simulated time per call
        dict(name="disk_1k_fp64", call="step", dist="disk", n=1000, form="fp64", behavior="elastic", cycles=20,
             dt=0.005),
        # the parity workload: a Plummer sphere in the plain form
        dict(name="plummer_16k_fp64", call="step", dist="plummer", n=16384, form="fp64", behavior="elastic", cycles=2,
             dt=0.01),
        # a parameter sweep of small collections in the plain form
        dict(name="batch_fp64", call="step", dist="ensemble", n=40, lo=256, hi=2048, form="fp64", behavior="mixed",
             cycles=4, dt=0.005),
        # interactive use of the fast form: a few thousand bodies, odd count
        dict(name="plummer_2k_mixed", call="step", dist="plummer", n=2501, form="mixed", behavior="elastic", cycles=20,
             dt=0.001),
        # an ordinary galaxy model, merging bodies, odd count
        dict(name="plummer_20k_mixed", call="step", dist="plummer", n=20011, form="mixed", behavior="subsume", cycles=5,
             dt=0.001),
        # the benchmark's headline collection; a run this long is tuned once
        dict(name="plummer_disk_131k_mixed", call="step", dist="plummer_disk", n=131072, form="mixed",
             behavior="subsume", cycles=3, dt=0.001, tune=True),
        # the largest direct sum, one cycle, as it comes (tuning it would take
        # longer than the run)
        dict(name="uniform_1m_mixed", call="step", dist="uniform", n=1048576, form="mixed", behavior="none", cycles=1,
             dt=0.001),
        # the benchmark's batch: 512 collections of 256 to 32,768 bodies
        dict(name="ensemble_512_mixed", call="step", dist="ensemble", n=512, lo=256, hi=32768, form="mixed",
             behavior="mixed", cycles=3, dt=0.001),
        # the octree at the headline size
        dict(name="plummer_131k_bh_mixed", call="step", dist="plummer", n=131072, form="mixed", bh=True,
             behavior="subsume", cycles=3, dt=0.001),
        # the octree where the direct sum is out of reach, ragged count
        dict(name="uniform_1m_bh_mixed", call="step", dist="uniform", n=1000003, form="mixed", bh=True,
             behavior="none", cycles=2, dt=0.001),
        # the reference's default force path in its own arithmetic
        dict(name="plummer_30k_bh_fp64", call="step", dist="plummer", n=30011, form="fp64", bh=True,
             behavior="elastic", cycles=1, dt=0.01),
        # the forces alone, for a caller with its own integrator
        dict(name="forces_50k_mixed", call="forces", dist="plummer", n=50001, form="mixed", behavior="none"),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["fp64", "mixed", "mixed", "batch_fp64", "batch_mixed", "bh_mixed", "bh_fp64", "forces"])
    # the plain form's workloads use 5 and 10 ms; the fast form is run finer
    dt = rng.choice([0.005, 0.01]) if "fp64" in kind else rng.choice([0.0005, 0.001])
    behavior = rng.choice(["none", "elastic", "subsume"])
    if kind == "fp64":
        n = _log_int(rng, 200, 20000)
        return dict(call="step", dist=rng.choice(["disk", "plummer"]), n=n, form="fp64", behavior=behavior,
                    cycles=max(1, min(20, int(6e8 / (n * n)))), dt=dt)
    if kind == "mixed":
        n = _log_int(rng, 500, 400000)
        return dict(call="step", dist=rng.choice(["disk", "plummer", "uniform"]), n=n, form="mixed", behavior=behavior,
                    cycles=max(1, min(20, int(5e10 / (n * n)))), dt=dt)
    if kind == "batch_fp64":
        return dict(call="step", dist="ensemble", n=rng.randint(3, 60), lo=200, hi=_log_int(rng, 600, 2500),
                    form="fp64", behavior="mixed", cycles=rng.randint(1, 4), dt=dt)
    if kind == "batch_mixed":
        return dict(call="step", dist="ensemble", n=_log_int(rng, 4, 500), lo=200, hi=_log_int(rng, 1000, 30000),
                    form="mixed", behavior="mixed", cycles=rng.randint(1, 3), dt=dt)
    if kind == "bh_mixed":
        n = _log_int(rng, 2000, 1000000)
        return dict(call="step", dist=rng.choice(["plummer", "uniform"]), n=n, form="mixed", bh=True,
                    behavior=behavior, cycles=rng.randint(1, 3), dt=dt)
    if kind == "bh_fp64":
        return dict(call="step", dist=rng.choice(["disk", "plummer"]), n=_log_int(rng, 1000, 40000), form="fp64",
                    bh=True, behavior=behavior, cycles=1, dt=dt)
    return dict(call="forces", dist=rng.choice(["disk", "plummer"]), n=_log_int(rng, 1000, 150000), form="mixed",
                behavior="none")


def _member(k, n, seed):
    """Collection k of a batch: the kinds, behaviours, masses and radii of
    workloads.ensemble."""
    behavior = (A.NONE, A.ELASTIC, A.SUBSUME)[k % 3]
    kind = (k // 3) % 3
    if kind == 0:
        b = workloads.uniform_ball(n, seed=seed, R=5.0 * n ** (1.0 / 3.0), mass=1.0, radius=0.1, behavior=behavior)
    elif kind == 1:
        b = workloads.plummer(n, seed=seed, a=200.0, total_mass=1e16, behavior=behavior)
    else:
        b = workloads.disk(n, seed=seed, behavior=behavior)
    r = workloads.SplitMix64(seed + 5)
    b["mass"][:] = r.log_uniform(n, 1e3, 1e6)
    b["radius"][:] = r.uniform(n, 0.1, 1.0)
    return b


def _bodies(case, seed):
    """The case's bodies (one dict of arrays) and the collections' counts."""
    n, s = case["n"], 1 + int(seed)
    if case["dist"] == "ensemble":
        # the sizes are the case's, the bodies the seed's
        counts = workloads.ensemble_sizes(n, 5, case["lo"], case["hi"])
        sims = [_member(k, int(c), s * 100003 + k) for k, c in enumerate(counts)]
        b = {k: np.concatenate([q[k] for q in sims]) for k in sims[0]}
        b["id"] = np.arange(len(b["x"]), dtype=np.int64)
        return b, counts
    if case["dist"] == "plummer_disk":
        b = workloads.plummer_disk(n // 2, seed=s)
    elif case["dist"] == "disk":
        b = workloads.disk(n, seed=s)
    elif case["dist"] == "uniform":
        b = workloads.uniform_ball(n, seed=s)
    else:
        b = workloads.plummer(n, seed=s)
    b["collision"][:] = BEHAVIOR[case["behavior"]]
    return b, np.array([len(b["x"])], dtype=np.int64)


def _pinned(n, dtype):
    dt = np.dtype(dtype)
    return torch.empty(max(1, n * dt.itemsize), dtype=torch.uint8, pin_memory=True).numpy()[:n * dt.itemsize].view(dt)


def prepare(case, seed):
    b, counts = _bodies(case, seed)
    n = int(counts.sum())
    bodies = {}
    for k, v in b.items():
        bodies[k] = _pinned(n, v.dtype)
        bodies[k][:] = v
    sim = Simulation(case["form"], capacity=n + 1)
    if case.get("bh"):
        sim.set_option(A.OPT_BARNES_HUT, 1)
    state = dict(case=case, sim=sim, bodies=bodies, counts=counts, shape=None)
    if case.get("tune"):
        _load(state)
        state["shape"] = sim.autotune()[0]
    if case["call"] == "step":
        fields = STATE + (FORCES if case["form"] == "fp64" else ())
        state["out"] = {f: _pinned(n, A.FIELD_DTYPES[f]) for f in fields}
        for v in state["out"].values():
            v[:] = 0
    return state


def _load(state):
    if len(state["counts"]) > 1:
        state["sim"].set_collections_flat(state["bodies"], state["counts"])
    else:
        state["sim"].set_bodies(state["bodies"])


def run(state):
    case, sim = state["case"], state["sim"]
    _load(state)
    if case["call"] == "forces":
        f = sim.force_pass()
        return {k: v.astype(np.float32) for k, v in zip(FORCES, f)}
    sim.step(case["dt"], 1.0, nsteps=case["cycles"])
    # the arrays of the program, as long as the collection was before bodies
    # merged; what a merge freed at their end stays as it was
    now = sim.state(out=state["out"])
    counts = sim.sim_counts() if len(state["counts"]) > 1 else len(now["x"])
    return dict(state["out"], counts=counts)


def work(case):
    if case["dist"] == "ensemble":
        counts = workloads.ensemble_sizes(case["n"], 5, case["lo"], case["hi"]).astype(float)
        n, pairs = counts.sum(), (counts * (counts - 1.0)).sum()
    else:
        n = case["n"]
        pairs = n * (n - 1.0)
    if case.get("bh"):
        # point-mass terms of the opening angle 0.3, about 28 / theta^2 per
        # e-folding of the body count (5,190 a body counted at 131,072, 3,600
        # at 2^20 uniform), never more than the direct sum's
        pairs = min(pairs, n * 310.0 * math.log(max(n, 2)))
    cycles = case.get("cycles", 1)
    # 20 flops a pair, the usual count of a gravity interaction; bytes: the
    # loaded fields (11 of 8 bytes, 2 of 4), the returned ones, and per cycle
    # the state a step reads and writes (position, velocity, mass, radius)
    back = 3 * 4 if case["call"] == "forces" else 9 * 8 + 4 + (24 if case["form"] == "fp64" else 0)
    return {"bytes": n * (11 * 8 + 2 * 4 + back + cycles * (8 + 6) * 8.0), "flops": 20.0 * pairs * cycles}


def _forces64(x, m, rad, live):
    """Forces of every live body on every other, FP64, with the overlap rule:
    pairs with dist <= r_i + r_j exert none and are returned as events."""
    n = x.shape[1]
    f = torch.zeros_like(x)
    events = []
    step = max(1, int(1.6e8) // max(1, n))
    for i0 in range(0, n, step):
        i1 = min(n, i0 + step)
        d = [x[c][None, :] - x[c][i0:i1, None] for c in range(3)]
        r2 = d[0] * d[0]
        r2.addcmul_(d[1], d[1]).addcmul_(d[2], d[2])
        dist = r2.sqrt_()
        hit = dist <= rad[i0:i1, None] + rad[None, :]
        hit &= live[i0:i1, None] & live[None, :]
        hit[torch.arange(i1 - i0), torch.arange(i0, i1)] = False
        w = (m * live)[None, :] / (dist * dist * dist)
        w[torch.arange(i1 - i0), torch.arange(i0, i1)] = 0.0
        w[hit] = 0.0
        for c in range(3):
            f[c, i0:i1] = (w * d[c]).sum(1)
        q = hit.nonzero()
        if len(q):
            events.append(torch.cat([q + torch.tensor([[i0, 0]], device=q.device), dist[hit][:, None]], 1))
    f *= G * m
    return f, events


def exact(case, seed):
    """The cycle in torch FP64: direct sum, merging (subsume) in the
    reference's order, symplectic Euler.  None where an elastic collision is
    met, for the octree (whose result is an approximation by its tree) and for
    sums of more than 1e11 pairs."""
    if case.get("bh") or case["dist"] == "ensemble":
        return None
    cycles = case.get("cycles", 1)
    if float(case["n"]) ** 2 * cycles > 1e11:
        return None
    b, _ = _bodies(case, seed)
    dev = torch.device("cuda", 0)
    x = torch.from_numpy(np.stack([b["x"], b["y"], b["z"]])).to(dev)
    v = torch.from_numpy(np.stack([b["vx"], b["vy"], b["vz"]])).to(dev)
    m, rad = torch.from_numpy(b["mass"]).to(dev), torch.from_numpy(b["radius"]).to(dev)
    f = torch.zeros_like(x)
    for _ in range(cycles):
        live = torch.ones_like(m, dtype=torch.bool)
        f, events = _forces64(x, m, rad, live)
        if events and case["call"] == "step":
            if case["behavior"] == "elastic":
                return None
            if case["behavior"] == "subsume":
                ev = torch.cat(events).cpu().numpy()
                mh, rh = m.cpu().numpy(), rad.cpu().numpy()
                keep = np.ones(len(mh), dtype=bool)
                for i, j, dist in ev[np.lexsort((ev[:, 1], ev[:, 0]))][::-1]:
                    i, j = int(i), int(j)
                    if rh[i] > rh[j] and dist <= rh[i]:
                        a, o = i, j
                    elif rh[j] > rh[i] and dist <= rh[j]:
                        a, o = j, i
                    else:
                        continue
                    mh[a] += mh[o]
                    mh[o] = 0.0
                    keep[o] = False
                m, live = torch.from_numpy(mh).to(dev), torch.from_numpy(keep).to(dev)
        if case["call"] == "forces":
            return dict(zip(FORCES, f))
        v = v + case["dt"] * f / m
        x = x + case["dt"] * v
        x, v, f = x[:, live], v[:, live], f[:, live]
        m, rad = m[live], rad[live]
    out = dict(x=x[0], y=x[1], z=x[2], vx=v[0], vy=v[1], vz=v[2], mass=m, radius=rad)
    if case["form"] == "fp64":
        out.update(zip(FORCES, f))
    whole = {k: torch.zeros(case["n"], dtype=torch.float64, device=dev) for k in out}
    for k, t in out.items():
        whole[k][:len(t)] = t
    return dict(whole, id=None, flags=None, counts=None)
