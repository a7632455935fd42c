"""The calls a user of the engine times: walks, batches, gradients, contractions.

Every case is one pass through the public entry points (``engine.Sim``,
``engine.batch_run``, ``engine.Graph``, ``engine.contract_phases``,
``adjoint.waveform_signal``), with the lattice shapes, time steps, record
counts and gradient tables that the benchmark, the tests and the simulator's
demo use.  Inputs are synthetic and made from a seed alone.
"""
from __future__ import annotations

import math
import random

import numpy as np
import torch

from rms_b200 import adjoint, analysis, engine, geometry, waveforms

DT = 2e-4                       # ms, the demo's time step
RES = 0.1                       # um, the voxel size of every lattice here
OPS_PER_WALKER_STEP = 105.0     # algorithmic thread-operations of one step of one walker


def _walk(name, **kw):
    """A walk: lattice (side, side, length), labels 1 in the axon and
    ``exterior`` outside (0: none, 2: extra-axonal water)."""
    case = dict(kind="walk", precision="split", side=64, length=512, exterior=2, walkers=100_000, steps=5000,
                records=1000, mode="moments", signals=0, boundary="mirror", kappa=-1.0, reload=False)
    case.update(kw)
    return dict(case, name=name) if name else case


def listed():
    return [
        # the demo's program as it comes: 1e3 walkers, FP64 in the reference's
        # order (the default precision), 1000 records, a 90-entry b-table
        _walk("demo 1e3 walkers, compat", precision="compat", walkers=1000, steps=2000, mode="narrow", signals=90),
        # the same small job in split precision with finite pulses: what a user
        # calls many times while setting a protocol up (latency)
        _walk("small PGSE, split", walkers=1000, steps=5000, mode="pgse", signals=60),
        # one FP64 run of a usual size: the plain form every split run is held to
        _walk("1e5 walkers, compat", precision="compat", steps=2000, mode="narrow", signals=12),
        # the single-axon benchmark: impermeable axon, moments every 10 steps
        _walk("single axon, split", exterior=0, records=500, boundary="periodic"),
        # narrow pulses with the full 90-entry b-table, an odd walker count
        _walk("b-table of 90, split", walkers=200_003, steps=4000, mode="narrow", signals=90),
        # the production job, fewer walkers and steps: large lattice,
        # permeable membrane, 540 PGSE gradients
        _walk("production PGSE, split", side=256, length=2048, walkers=1_000_000, steps=4000, mode="pgse",
              signals=540, kappa=0.01),
        # a study's next lattice handed to a simulation that has run, then a walk
        _walk("new lattice, then walk", side=128, length=1024, walkers=50_000, steps=1000, reload=True),
        # many axons of uneven lattices in one captured launch
        dict(name="16 axons, graph", kind="batch", axons=16, graph=True, lo=64, hi=192, long_lo=256, long_hi=1536,
             walkers=4_000_000, steps=2000, records=1000, even=False),
        # the demo's study: many axons with 1e3 walkers each
        dict(name="64 axons of 1e3 walkers", kind="batch", axons=64, graph=False, lo=48, hi=96, long_lo=200,
             long_hi=400, walkers=64_000, steps=2000, records=1000, even=True),
        # fitting waveforms: the signal and its gradients through torch
        dict(name="waveform gradients", kind="gradient", how="backward", side=64, length=512, walkers=100_000,
             steps=5000, bins=1000, waves=16),
        # phases of many waveforms from trajectories already on the GPU
        dict(name="1024 waveforms, 1e6 walkers", kind="contract", method="bf16x3", walkers=1_000_000, bins=256,
             waves=1024),
        # a walk that leaves split trajectories and their contraction
        dict(name="walk and contraction", kind="trajectory", side=64, length=512, walkers=100_000, steps=1280,
             bins=256, waves=512),
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng: random.Random) -> dict:
    kind = rng.choice(["walk", "walk", "walk", "walk", "batch", "gradient", "contract", "trajectory"])
    if kind == "walk":
        precision = rng.choice(["compat", "split", "split"])
        steps = int(_log(rng, 1000, 8000))
        most = 3e8 if precision == "compat" else 3e9
        walkers = int(_log(rng, 500, min(1_000_000, most / steps)))
        mode = rng.choice(["moments", "narrow", "pgse"])
        reload = rng.random() < 0.2
        side = int(_log(rng, 40, 128 if reload else 256))
        return _walk(None, precision=precision, side=side, length=int(side * rng.uniform(3, 8)),
                     exterior=rng.choice([0, 2, 2]), walkers=walkers, steps=steps,
                     records=rng.choice([1000, 1000, 500, 200, 100]), mode=mode,
                     signals={"moments": 0, "narrow": rng.randint(1, 90), "pgse": int(_log(rng, 6, 540))}[mode],
                     boundary=rng.choice(["mirror", "mirror", "periodic"]),
                     kappa=rng.choice([-1.0, 0.01, 0.05]), reload=reload)
    if kind == "batch":
        axons, even = int(_log(rng, 4, 64)), rng.random() < 0.5
        lo = rng.randint(40, 64)
        return dict(kind=kind, axons=axons, graph=rng.random() < 0.5, lo=lo, hi=rng.randint(lo, 144),
                    long_lo=rng.randint(200, 300), long_hi=rng.randint(300, 1024),
                    walkers=axons * int(_log(rng, 500, 60_000)), steps=int(_log(rng, 1000, 2000)),
                    records=rng.choice([1000, 500, 200]), even=even)
    if kind == "gradient":
        bins = rng.choice([100, 250, 500, 1000])
        return dict(kind=kind, how=rng.choice(["backward", "jacobian"]), side=rng.randint(48, 80),
                    length=rng.randint(300, 600), walkers=int(_log(rng, 2000, 100_000)),
                    steps=bins * rng.randint(-(-1000 // bins), 5000 // bins), bins=bins, waves=rng.randint(1, 16))
    if kind == "contract":
        return dict(kind=kind, method=rng.choice(["bf16x3", "bf16x3", "fp32"]), walkers=int(_log(rng, 4000, 300_000)),
                    bins=4 * rng.randint(8, 64), waves=int(_log(rng, 16, 1024)))
    bins = 8 * rng.randint(8, 32)
    return dict(kind=kind, side=rng.randint(48, 80), length=rng.randint(300, 600),
                walkers=int(_log(rng, 4000, 100_000)), steps=bins * rng.randint(4, 8), bins=bins,
                waves=int(_log(rng, 32, 512)))


# ---------------------------------------------------------------------------
# what a user's program holds before the call

def _directions(rng, n):
    v = rng.normal(size=(n, 3))
    return v / np.linalg.norm(v, axis=1, keepdims=True)


def _b_table(rng, n):
    """n b-values (ms/um^2) on four shells, each with its own direction."""
    return rng.choice([0.5, 1.0, 1.5, 2.0], size=n), _directions(rng, n)


def _pgse_table(rng, n, total):
    """n gradients: Delta on three values, delta a quarter of the walk, b in 0..5."""
    delta = 0.25 * total
    rows = []
    for j, d in enumerate(_directions(rng, n)):
        Delta = total * (0.5, 0.6, 0.7)[j % 3]
        rows.append([Delta, delta, float(analysis.pgse_gradient_for_b(float((j // 3) % 6), Delta, delta)), *d])
    return np.array(rows)


def _walk_state(case, seed):
    rng = np.random.default_rng(seed)
    side, length = case["side"], case["length"]
    kw = dict(dt=DT, tn=case["steps"], npar=case["walkers"], res=RES,
              diffusivity=[0.0, 2.0, 2.0 if case["kappa"] >= 0 else 1.5], t2=[80.0, 80.0, 60.0], shape=(side, side, length),
              timepoints=case["records"], boundary=case["boundary"])
    if case["kappa"] >= 0:
        kw.update(permeation="kappa", kappa=case["kappa"])
    if case["mode"] == "pgse":
        kw["grad"] = _pgse_table(rng, case["signals"], case["steps"] * DT)
    elif case["mode"] == "narrow":
        kw["bval"], kw["bvec"] = _b_table(rng, case["signals"])
    sim = engine.Sim(**kw)
    state = dict(sim=sim, seed=seed, precision=case["precision"], labels=None)
    if case["reload"]:
        state["labels"] = geometry.axon_lattice(side, side, length, RES, seed, exterior=case["exterior"])
    if state["labels"] is None:
        sim.set_tube_lattice(*geometry.axon_slices(side, side, length, RES, seed), inside=1, outside=case["exterior"])
    else:
        # the simulation has run before: it has its device
        sim.set_lattice(state["labels"])
        sim.run(seed=seed, precision=case["precision"], walker_range=(0, min(32, case["walkers"])))
    return state


def _batch_state(case, seed):
    rng = np.random.default_rng(seed)
    shapes = geometry.batch_sizes(case["axons"], seed, lo=(case["lo"], case["lo"], case["long_lo"]),
                                  hi=(case["hi"], case["hi"], case["long_hi"]))
    tubes = [geometry.axon_slices(*s, RES, seed + k) for k, s in enumerate(shapes)]
    volume = np.array([1.0 if case["even"] else r2.sum() for r2, _, _ in tubes])
    npar = np.maximum(32, case["walkers"] * volume / volume.sum()).astype(int)
    sims = []
    for shape, tube, n in zip(shapes, tubes, npar):
        D = float(rng.uniform(1.5, 2.5))
        sim = engine.Sim(dt=DT, tn=case["steps"], npar=int(n), res=RES, diffusivity=[0.0, D, D], t2=[80.0, 80.0, 60.0],
                         shape=shape, timepoints=case["records"], permeation="kappa",
                         kappa=float(rng.uniform(0.0, 0.05)))
        sim.set_tube_lattice(*tube, inside=1, outside=2)
        sims.append(sim)
    graph = engine.Graph(sims, seed=seed) if case["graph"] else None
    return dict(sims=sims, graph=graph, seed=seed)


def _smooth_waves(n, bins, total, seed, bmax):
    """n smooth waveforms [n, bins, 3] with b-values up to bmax, phase per um per ms."""
    w = waveforms.random_smooth(n, bins, 1.0, seed=seed)
    return np.ascontiguousarray(waveforms.scale_to_b(w, total / bins, np.linspace(0.1, bmax, n)))


def _gradient_state(case, seed):
    labels = geometry.axon_lattice(case["side"], case["side"], case["length"], RES, seed, exterior=2)
    wave = _smooth_waves(case["waves"], case["bins"], case["steps"] * DT, seed, 4.0)
    setup = adjoint.WalkSetup(labels, dt=DT, tn=case["steps"], npar=case["walkers"], res=RES, seed=seed,
                              boundary="periodic")
    rng = np.random.default_rng(seed)
    return dict(setup=setup, wave=torch.tensor(wave, dtype=torch.float32), D=torch.tensor(2.0),
                kappa=torch.tensor(0.02), t2=torch.tensor([80.0, 80.0, 60.0]),
                weights=torch.tensor(rng.normal(size=(case["waves"], 2)), dtype=torch.float32))


def _contract_state(case, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    bin_time = 10.0 / case["bins"]
    pos = torch.empty((case["walkers"], case["bins"], 3), dtype=torch.float32, device="cuda")
    pos.normal_(std=math.sqrt(2.0 * 2.0 * bin_time), generator=g)
    pos = torch.cumsum(pos, dim=1).contiguous()
    wave = _smooth_waves(case["waves"], case["bins"], 10.0, seed, 10.0) * bin_time
    return dict(pos=pos, wave=torch.tensor(wave, dtype=torch.float32, device="cuda"),
                out=torch.empty((case["waves"], 2), dtype=torch.float64, device="cuda"))


def _trajectory_state(case, seed):
    total = case["steps"] * DT
    sim = engine.Sim(dt=DT, tn=case["steps"], npar=case["walkers"], res=RES, diffusivity=[0.0, 2.0, 2.0],
                     t2=[80.0, 80.0, 60.0], shape=(case["side"], case["side"], case["length"]),
                     wave=np.zeros((1, case["bins"], 3)), timepoints=case["bins"], boundary="periodic")
    sim.set_tube_lattice(*geometry.axon_slices(case["side"], case["side"], case["length"], RES, seed), inside=1,
                         outside=2)
    wave = _smooth_waves(case["waves"], case["bins"], total, seed, 4.0) * (total / case["bins"])
    return dict(sim=sim, seed=seed, wave=torch.tensor(wave, dtype=torch.float32, device="cuda"),
                traj=torch.empty((case["walkers"], case["bins"], 3), dtype=torch.float32, device="cuda"),
                out=torch.empty((case["waves"], 2), dtype=torch.float64, device="cuda"))


_PREPARE = dict(walk=_walk_state, batch=_batch_state, gradient=_gradient_state, contract=_contract_state,
                trajectory=_trajectory_state)


def prepare(case: dict, seed: int):
    return dict(_PREPARE[case["kind"]](case, seed), case=case)


# ---------------------------------------------------------------------------
# one pass

def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "walk":
        sim = state["sim"]
        if state["labels"] is not None:
            sim.set_lattice(state["labels"])
        return sim.run(seed=state["seed"], precision=state["precision"]).outputs()
    if kind == "batch":
        if state["graph"] is not None:
            state["graph"].run(state["seed"])
        else:
            engine.batch_run(state["sims"], seed=state["seed"], precision="split")
        rows = [s.outputs() for s in state["sims"]]
        return {k: np.stack([r[k] for r in rows]) for k in ("sig0", "dx2", "dx4", "npar_count")}
    if kind == "gradient":
        if case["how"] == "jacobian":
            return adjoint.signal_jacobian(state["wave"], state["D"], state["kappa"], state["t2"], state["setup"])
        leaves = [state[k].detach().clone().requires_grad_(True) for k in ("wave", "D", "kappa", "t2")]
        signal = adjoint.waveform_signal(*leaves, state["setup"])
        (signal * state["weights"]).sum().backward()
        return dict(signal=signal.detach(), **{k: x.grad for k, x in zip(("wave", "D", "kappa", "t2"), leaves)})
    out = state["out"]
    if kind == "contract":
        pos, method = state["pos"], case["method"]
    else:
        pos, method = state["traj"], "bf16x3_presplit"
        state["sim"].run(seed=state["seed"], precision="split", traj_out=pos.data_ptr(), traj_split=True)
    engine.contract_phases(pos.data_ptr(), case["walkers"], case["bins"], state["wave"].data_ptr(), case["waves"],
                           out.data_ptr(), method=method, stream=torch.cuda.current_stream().cuda_stream)
    if kind == "contract":
        return out
    return dict(sums=out, walk=state["sim"].outputs())


def exact(case: dict, seed: int):
    """64-bit sums of the contraction; the walks are Monte Carlo sums over
    FP32 or FP64 trajectories with no closed value."""
    if case["kind"] != "contract":
        return None
    state = _contract_state(case, seed)
    K = case["bins"] * 3
    pos, wave = state["pos"].view(-1, K), state["wave"].view(-1, K).double()
    total = torch.zeros((case["waves"], 2), dtype=torch.float64, device="cuda")
    for part in pos.split(65536):
        phase = part.double() @ wave.T
        total[:, 0] += phase.cos().sum(0)
        total[:, 1] += phase.sin().sum(0)
    return total


# ---------------------------------------------------------------------------
# work a pass cannot do without

def work(case: dict) -> dict:
    kind = case["kind"]
    n = case["walkers"]
    if kind == "contract":
        K = 3 * case["bins"]
        return dict(bytes=4.0 * K * (n + case["waves"]) + 16.0 * case["waves"], flops=2.0 * n * K * case["waves"])
    flops = OPS_PER_WALKER_STEP * n * case["steps"]
    if kind == "batch":
        side, length = (case["lo"] + case["hi"]) / 2, (case["long_lo"] + case["long_hi"]) / 2
        return dict(bytes=case["axons"] * (side * side * length + 8.0 * 25 * case["records"]), flops=flops)
    voxels = float(case["side"]) ** 2 * case["length"]
    if kind == "walk":
        narrow = case["signals"] if case["mode"] == "narrow" else 0
        out = 8.0 * (case["records"] * (25 + narrow) + case["signals"])
        signal_ops = 8.0 * n * (case["records"] * narrow + (case["signals"] if case["mode"] == "pgse" else 0))
        return dict(bytes=voxels + out, flops=flops + signal_ops)
    if kind == "gradient":
        phase_ops = 12.0 * n * case["bins"] * case["waves"]
        walks = 1.0 if case["how"] == "jacobian" else 2.0
        return dict(bytes=voxels + 8.0 * 3 * case["bins"] * case["waves"], flops=walks * (flops + phase_ops))
    K = 3 * case["bins"]
    return dict(bytes=voxels + 2 * 4.0 * K * n + 4.0 * K * case["waves"], flops=flops + 2.0 * n * K * case["waves"])
