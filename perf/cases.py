"""Workloads of the sampler and of its warm-start generator, for timing and comparing builds.

Every case goes through the package's public classes, as a program that uses them would. The
sizes are those of the benchmark's configurations, of the tests, or generic ones between them.
The chains of a case are random starts swept for a while in prepare(), so that a pass meets the
acceptance rates of a running simulation. Samples are kept as float32, the type of the protocol
driver's datasets (mags.npy, energies.npy, top_chars.npy, ...).
"""
from __future__ import annotations

import math

import numpy as np

from nanomagmc_gb300 import _lib as L
from nanomagmc_gb300.sampler import Sampler, interactions_file, make_options, read_interactions
from nanomagmc_gb300.warmstart import Generator, heisenberg_sampler

# kind "step":    one sample step, sweeps then every observable (nmmc_sweep_measure)
# kind "series":  several sample steps from one call (nmmc_sample)
# kind "point":   one (T, H) point of the protocol driver: fork, parameters, equilibration,
#                 samples with a summed lattice, and the lattices it prints
# kind "observe": observables of given lattices (nmmc_measure)
# kind "warm":    learned warm start of a batch of chains, and their observables
# kind "train":   one training step of the generator, with its gradients
CHAIN = dict(kind="step", shape="s", edge=64, mean=0.0, dev=0.0, ising=False, periodic=True,
             table="2d_nn_interfacial.dat", dmi=0.5, chains=1, t0=0.05, t1=1.5, h0=0.0, h1=0.0,
             sweeps=10, samples=1, settle=30)


def _chains(name, **kw):
    return dict(CHAIN, name=name, **kw)


def listed():
    return [
        # the smallest call: the benchmark's 2-D Ising scan around its transition, a launch or
        # two per sample
        _chains("ising2d_32", edge=32, ising=True, table="2d_nn.dat", dmi=0.0, chains=13, t0=2.0, t1=2.6),
        # a skyrmion phase diagram: one chain per (B, T) point (the benchmark's 21 x 20 grid)
        _chains("heis2d_64_grid", edge=64, chains=420, h1=1.0, sweeps=20),
        # log-normal Weibull grains, open and ragged, 1-2 thousand sites each (512, radius 20)
        _chains("grains_512", shape="w", edge=90, mean=20.0, dev=5.0, periodic=False, chains=512, h1=1.0),
        # the benchmark workload, and the largest case: 40 temperatures of a 128^3 cube
        _chains("heis3d_128", shape="c", edge=128, table="3d_nn_bloch.dat", dmi=0.3, chains=40, t0=0.2, t1=2.0,
                h0=0.2, h1=0.2, settle=10),
        # a batch of 16 large 2-D lattices sampled in series, as after a warm start
        _chains("heis2d_128_series", kind="series", edge=128, chains=16, t0=0.3, t1=0.9, h0=0.25, h1=0.25,
                sweeps=20, samples=5),
        # an interaction file beyond nearest neighbours (J1 + 12 face-diagonal J2, bulk DMI)
        _chains("j1j2_64", shape="c", edge=64, table="3d_j1j2_bloch.dat", dmi=0.3, chains=20, t0=0.2, t1=2.0,
                h0=0.2, h1=0.2),
        # 3-D Weibull particles, too large for one SM (the benchmark's radius 30 in 90^3 boxes)
        _chains("spheres_30", shape="x", edge=90, mean=30.0, periodic=False, table="3d_nn_bloch.dat", dmi=0.3,
                chains=24, t0=0.2, t1=2.0, h0=0.2, h1=0.2),
        # 3-D Ising around its transition (T = 4.51): finite-size scaling runs
        _chains("ising3d_64", shape="c", edge=64, ising=True, table="3d_nn_bloch.dat", dmi=0.0, chains=24,
                t0=4.0, t1=5.0),
        # one inner point of the protocol driver on 8 small cubes whose rows are no multiple of a
        # vector (15 sites per colour), with its printed lattices
        _chains("point_30", kind="point", shape="c", edge=30, table="3d_nn_bloch.dat", dmi=0.3, chains=8, t0=0.6,
                t1=1.4, h0=0.2, h1=0.2, sweeps=10, samples=5, settle=50),
        # observables alone, of open cubes of an odd edge (State.energy(), magnetisation(), ...)
        _chains("observe_33", kind="observe", shape="c", edge=33, periodic=False, table="3d_nn_bloch.dat", dmi=0.3,
                chains=32, t0=0.5, t1=2.0, h0=0.1, h1=0.4, settle=0),
        # learned warm start of 16 lattices, the benchmark's 8 denoising passes
        dict(name="warm_128", kind="warm", edge=128, chains=16, passes=8),
        # one training step of the generator at the benchmark's batch of 16
        dict(name="train_128", kind="train", edge=128, batch=16, snapshots=64),
    ]


def _log(rng, a, b):
    return math.exp(rng.uniform(math.log(a), math.log(b)))


def draw(rng):
    pick = rng.randrange(12)
    if pick == 0:   # 2-D Ising, periodic (even) or open
        per = rng.random() < 0.6
        edge = int(_log(rng, 12, 200))
        edge += (edge & 1) if per else 0
        return dict(CHAIN, edge=edge, ising=True, table="2d_nn.dat", dmi=0.0, periodic=per,
                    chains=int(_log(rng, 1, 64)), t0=1.8, t1=2.8, sweeps=rng.choice([5, 10, 20]))
    if pick in (1, 2):   # 2-D Heisenberg
        per = rng.random() < 0.7
        edge = int(_log(rng, 16, 160))
        edge += (edge & 1) if per else 0
        most = max(2, min(500, 1700000 // (edge * edge)))
        return dict(CHAIN, edge=edge, periodic=per, chains=int(_log(rng, 1, most)), h1=rng.choice([0.0, 0.5, 1.0]),
                    table=rng.choice(["2d_nn_interfacial.dat", "2d_nn_bloch.dat"]), sweeps=rng.choice([5, 10, 20]))
    if pick == 3:   # Weibull grains
        mean = round(_log(rng, 6, 30), 1)
        dev = round(mean * rng.uniform(0.1, 0.3), 1)
        return dict(CHAIN, shape="w", edge=int((mean + 2 * dev) * 3), mean=mean, dev=dev, periodic=False,
                    chains=int(_log(rng, 16, 500)), h1=1.0)
    if pick in (4, 5):   # cubes
        per = rng.random() < 0.7
        edge = int(_log(rng, 12, 128))
        edge += (edge & 1) if per else 0
        most = max(1, min(200, 40000000 // edge ** 3))
        return dict(CHAIN, shape="c", edge=edge, periodic=per, table="3d_nn_bloch.dat",
                    dmi=rng.choice([0.0, 0.3, 0.5]), chains=int(_log(rng, 1, most)), t0=0.2, t1=2.0, h0=0.0, h1=0.3,
                    settle=10)
    if pick == 6:   # general tables
        edge = 2 * int(_log(rng, 8, 32))
        return dict(CHAIN, shape="c", edge=edge, table="3d_j1j2_bloch.dat", dmi=0.3,
                    chains=int(_log(rng, 2, max(3, min(64, 5000000 // edge ** 3)))), t0=0.2, t1=2.0, h0=0.2, h1=0.2,
                    settle=10)
    if pick == 7:   # 3-D Weibull particles
        mean = round(_log(rng, 5, 30), 1)
        return dict(CHAIN, shape="x", edge=int(mean * 3), mean=mean, periodic=False, table="3d_nn_bloch.dat",
                    dmi=0.3, chains=int(_log(rng, 2, 24)), t0=0.2, t1=2.0, h0=0.2, h1=0.2, settle=10)
    if pick == 8:   # 3-D Ising
        per = rng.random() < 0.7
        edge = int(_log(rng, 12, 80))
        edge += (edge & 1) if per else 0
        return dict(CHAIN, shape="c", edge=edge, ising=True, periodic=per, table="3d_nn_bloch.dat", dmi=0.0,
                    chains=int(_log(rng, 1, max(2, min(64, 6000000 // edge ** 3)))), t0=4.0, t1=5.0)
    if pick == 9:   # series and protocol points
        if rng.random() < 0.5:
            edge = 2 * int(_log(rng, 16, 70))
            return dict(CHAIN, kind="series", edge=edge, chains=int(_log(rng, 2, 32)), t0=0.3, t1=0.9, h0=0.25,
                        h1=0.25, sweeps=rng.choice([5, 10, 20]), samples=rng.randrange(2, 8))
        edge = 2 * int(_log(rng, 8, 24))
        return dict(CHAIN, kind="point", shape="c", edge=edge, table="3d_nn_bloch.dat", dmi=0.3,
                    chains=rng.randrange(1, 9), t0=0.6, t1=1.4, h0=0.2, h1=0.2, samples=rng.randrange(2, 8),
                    settle=30)
    if pick == 10:   # observables
        edge = int(_log(rng, 12, 50))
        per = edge % 2 == 0 and rng.random() < 0.5
        return dict(CHAIN, kind="observe", shape="c", edge=edge, periodic=per, table="3d_nn_bloch.dat",
                    dmi=rng.choice([0.0, 0.3]), chains=int(_log(rng, 1, 48)), t0=0.5, t1=2.0, h0=0.1, h1=0.4,
                    settle=0)
    if rng.random() < 0.5:   # generator
        return dict(kind="warm", edge=rng.choice([32, 64, 128]), chains=rng.randrange(1, 17), passes=rng.randrange(2, 9))
    return dict(kind="train", edge=rng.choice([32, 64, 128]), batch=rng.randrange(1, 17), snapshots=64)


# ------------------------------------------------------------------------------------------
# inputs
# ------------------------------------------------------------------------------------------
def _dim(case):
    return 3 if case["shape"] in "cx" else 2


def _points(case, n, seed=None):
    """n (T, H) points of a grid over the case's ranges; with a seed, each T moved by up to 5 %."""
    rows = max(1, int(math.sqrt(n))) if case["h1"] > case["h0"] else 1
    cols = -(-n // rows)
    T, H = np.meshgrid(np.linspace(case["t0"], case["t1"], cols), np.linspace(case["h0"], case["h1"], rows))
    T, H = T.ravel()[:n], H.ravel()[:n]
    if seed is not None:
        T = T * np.random.default_rng(seed).uniform(0.95, 1.05, n)
    return T, H


def _sampler(case, seed, copies=1):
    n = case["chains"]
    opt = make_options(case["shape"], edge=case["edge"], size=case["mean"] or None, ising=case["ising"],
                       periodic=case["periodic"], J=1.0, D=case["dmi"], weibull=3.0, asd=case["dev"])
    inter = read_interactions(interactions_file(case["table"]), _dim(case), 1.0, case["dmi"])
    sizes = None
    if case["dev"]:
        m, d = case["mean"], case["dev"]
        lm, ls = math.log(m * m / math.sqrt(d * d + m * m)), math.sqrt(math.log(1 + d * d / (m * m)))
        sizes = [L.load().nmmc_lognormal_size(7, k, lm, ls) for k in range(n)]
    # Weibull shapes: one set of particles (drawn from the sampler's seed) at points that differ
    # with the case's seed; other lattices: other random streams
    weibull = case["shape"] in "wx"
    T, H = _points(case, n, seed if weibull else None)
    return Sampler(opt, inter, T=np.tile(T, copies), H=np.tile(H, copies), sizes=sizes,
                   lattices=np.tile(np.arange(n), copies), seed=1000 if weibull else seed + 1)


def _given_spins(case, seed):
    """Unit vectors in FP32 precision, partly aligned along +z, per chain in box order."""
    rng = np.random.default_rng(seed)
    v = rng.standard_normal((case["chains"], case["edge"] ** 3, 3)) + np.array([0.0, 0.0, 0.5])
    v /= np.linalg.norm(v, axis=2, keepdims=True)
    return v.astype(np.float32).astype(np.float64)


def prepare(case, seed):
    if case["kind"] in ("warm", "train"):
        n = case["chains"] if case["kind"] == "warm" else 16
        rng = np.random.default_rng(seed)
        T, B = rng.uniform(0.3, 1.5, n), rng.uniform(0.0, 1.0, n)
        s = heisenberg_sampler(case["edge"], 0.5, T, B, seed=seed + 1)
        gen = Generator(case["edge"], capacity=case.get("snapshots", 0), seed=seed + 2)
        cond = np.stack([T, B, np.full(n, 0.5)], 1)
        if case["kind"] == "warm":
            return dict(case=case, s=s, gen=gen, chains=np.arange(n), cond=cond)
        for _ in range(case["snapshots"] // n):
            s.sweep(20)
            gen.add_snapshots(s, np.arange(n), cond)
        return dict(case=case, gen=gen, idx=rng.integers(0, gen.size, case["batch"]),
                    sig=np.clip(np.sqrt(rng.uniform(0.0, 1.0, case["batch"])), 0.02, 1.0))
    s = _sampler(case, seed, copies=2 if case["kind"] == "point" else 1)
    if case["kind"] == "observe":
        for k, v in enumerate(_given_spins(case, seed)):
            s.set_spins(k, v)
    elif case["kind"] == "point":
        s.sweep(case["settle"], np.arange(case["chains"]))
    else:
        s.sweep(case["settle"])
    s.synchronize()
    return dict(case=case, s=s)


# ------------------------------------------------------------------------------------------
# one pass
# ------------------------------------------------------------------------------------------
def _samples(obs, q):
    out = {"energy": obs[..., 0], "mag": obs[..., 1:5], "submag": obs[..., 5:9], "sub4mag": obs[..., 9:13],
           "charge": obs[..., 13], "slices": q}
    return {k: np.ascontiguousarray(v, np.float32) for k, v in out.items()}


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "train":
        loss = state["gen"].train_step(state["idx"], state["sig"], 1e-3)
        return {"loss": np.array([loss], np.float32), "grads": state["gen"].grads()}
    s = state["s"]
    if kind == "warm":
        state["gen"].warm_start(s, state["chains"], state["cond"], steps=case["passes"])
        out = _samples(*s.measure())
        out["lattice"] = s.get_spins(0)
        return out
    if kind == "step":
        return _samples(*s.sweep_measure(case["sweeps"], accumulate=True))
    if kind == "series":
        return _samples(*s.sample(case["sweeps"], case["samples"], with_q=True))
    if kind == "observe":
        return _samples(*s.measure())
    n = case["chains"]   # the protocol driver's inner loop over one (T, H) point
    T, H = _points(case, n)
    curr = np.arange(n, 2 * n)
    for k in range(n):
        s.fork(k, n + k)
    s.set_points(curr, T, H)
    s.sweep(case["settle"], curr)
    s.set_av_chains([n])
    out = _samples(*s.sample(case["sweeps"], case["samples"], curr, with_q=True))
    out["av_latt"] = s.get_av(n)
    out["sing_latt"] = s.get_spins(n)
    return out


# ------------------------------------------------------------------------------------------
# what a pass cannot do without
# ------------------------------------------------------------------------------------------
def _sites(case):
    """Filled sites of all chains (about, for Weibull shapes)."""
    e = case["edge"]
    if case["shape"] == "w":
        return int(case["chains"] * math.pi * (0.87 * case["mean"]) ** 2)
    if case["shape"] == "x":
        return int(case["chains"] * 4.19 * case["mean"] ** 3)
    return case["chains"] * e ** _dim(case)


def work(case):
    """Bytes: spins in and (where they change) out once, results once. Operations: per update
    the generator's 10 rounds (60 integer operations), the proposal and its test (about 30) and
    6 (J) or 18 (J and D) per neighbour; a tenth of that for an Ising neighbour. Observables:
    the bonds, 10 sums and two solid angles (about 80) per site. Convolutions: 2 per product."""
    if case["kind"] in ("warm", "train"):
        n = case["chains"] if case["kind"] == "warm" else case["batch"]
        px = n * case["edge"] ** 2
        macs = px * 9 * (8 * 48 + 6 * 48 * 48 + 48 * 4)
        if case["kind"] == "warm":
            return {"bytes": px * 24.0, "flops": 2.0 * macs * case["passes"]}
        return {"bytes": px * 12.0 + 4 * 9 * (8 * 48 + 6 * 48 * 48 + 48 * 4), "flops": 6.0 * macs}
    n, dim = _sites(case), _dim(case)
    nb = 18 if "j1j2" in case["table"] else 2 * dim
    spin = 1 if case["ising"] else 12
    update = 60 + (10 + 2 * nb if case["ising"] else 30 + (18 if case["dmi"] else 6) * nb)
    look = 4 + 2 * nb if case["ising"] else 10 + 80 + (18 if case["dmi"] else 6) * nb
    res = 8 * case["chains"] * (14 + (case["edge"] if dim == 3 else 1)) * case["samples"]
    if case["kind"] == "observe":
        return {"bytes": float(n * spin + res), "flops": float(n * look)}
    sweeps = case["sweeps"] * case["samples"]
    if case["kind"] == "point":
        sweeps += case["settle"]
        res += 48 * case["edge"] ** dim
    return {"bytes": float(2 * n * spin + res), "flops": float(n * (update * sweeps + look * case["samples"]))}


# ------------------------------------------------------------------------------------------
# 64-bit values of the observables (a Metropolis chain has none: its accepted moves are the
# result of FP32 tests, and the generator's layers round to BF16)
# ------------------------------------------------------------------------------------------
def exact(case, seed):
    if case["kind"] != "observe":
        return None
    e, n, per = case["edge"], case["chains"], case["periodic"]
    spins = _given_spins(case, seed).reshape(n, e, e, e, 3)   # [chain][z][y][x][component]
    _, H = _points(case, n)
    z, y, x = np.meshgrid(*(np.arange(e),) * 3, indexing="ij")
    sub = (x + y + z) % 2 == 0
    summ, diff = x + y, np.fmod(y - x + (e - e % 4), 4)   # C remainders
    sub4 = ((summ % 4 == 0) & (diff == 0) & (z % 4 == 0)) | ((summ % 4 == 2) & (diff == 2) & (z % 4 == 2))
    obs, q = np.zeros((n, 14)), np.zeros((n, e))

    def shifted(s, axis, step, wrap):   # the neighbour at +step along axis (0 where there is none)
        t = np.roll(s, -step, axis)
        if not wrap:
            edge = [slice(None)] * 4
            edge[axis] = -1 if step > 0 else 0
            t[tuple(edge)] = 0.0
        return t

    for k in range(n):
        s = spins[k]
        field = np.zeros_like(s)
        for axis, comp in ((2, 0), (1, 1), (0, 2)):
            for step in (1, -1):
                t = shifted(s, axis, step, per)
                d = np.zeros(3)
                d[comp] = step * case["dmi"]
                field += t + np.cross(d, t)
        m = s.reshape(-1, 3).sum(0)
        obs[k, 0] = -H[k] * m[2] - 0.5 * float((s * field).sum())
        for at, v in ((1, m), (5, s[sub].sum(0)), (9, s[sub4].sum(0))):
            obs[k, at:at + 3] = v
            obs[k, at + 3] = np.linalg.norm(v)
        for sx, sy in ((-1, 1), (1, -1)):   # triangles (i, i-x, i+y) and (i, i+x, i-y), never wrapped
            b, c = shifted(s, 2, sx, False), shifted(s, 1, sy, False)
            ok = ((x + sx >= 0) & (x + sx < e) & (y + sy >= 0) & (y + sy < e))
            dots = 1.0 + (s * b).sum(-1) + (s * c).sum(-1) + (b * c).sum(-1)
            ang = -np.arctan2((np.cross(s, c) * b).sum(-1), dots)
            q[k] += np.where(ok, ang, 0.0).sum((1, 2)) / (2 * math.pi)
        obs[k, 13] = q[k].sum()
    v = {"energy": obs[:, 0], "mag": obs[:, 1:5], "submag": obs[:, 5:9], "sub4mag": obs[:, 9:13],
         "charge": obs[:, 13], "slices": q}
    return v
