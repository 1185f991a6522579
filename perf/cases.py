"""Measured cases: the work that programs have this library do, through its public entry points.

Kinds of case (field "kind"):

  window    steps of one resident simulation, then the grain series of those steps and the ion
            state: what a run does between two file frames (OutputParameters.nFileOutput) and
            what a driver of short windows does. All-pairs or cutoff force, Maxwellian or
            field-driven plasma, every collision model and charge method.
  fork      one iteration of a dust-dynamics driver on the chains/matthews.py model: grains
            moved, a window of steps, series and state.
  batch     steps of several simulations resident in one batch, each with its own size, grains
            and force interval (a sweep, or a chunk of the request server).
  simulate  a whole OpenDust.simulate() call, set-up included.
  snapshot  the ion-ion force on a given snapshot (Engine.force_snapshot): analysis of frames,
            choice of a cutoff, tuning.
  static    od_ion_forces_static on the caller's own device arrays (plug-ins of other codes).

Sizes come from the named workloads (opendust_gb300.workloads), the tests and the benchmark:
2^11 .. 2^20 ions for windows, 2^14 .. 2^18 for sweep members, at most 2^15 for the static entry.

The engine computes ions in 32 bits and hands them out in float64 arrays; the cases keep ion
states, ion forces and the sums of ion terms on the grains as float32, as a program that stores
frames does. Charges and grain-grain forces are FP64 on the device and stay float64.
"""
from __future__ import annotations

import ctypes
import math
import random

import numpy as np
import torch

import opendust_gb300 as od
from opendust_gb300 import _lib, matthews, setup_host, workloads

# series rows of a window case: a run's series is long; a new window starts when it is full
SERIES_ROWS = 4096

METHODS = ("given", "consistent", "oml")


def listed():
    return [
        # smallest runs (smoke tests, parameter checks): launches and latency are the cost
        dict(name="window_tiny", kind="window", n=2048, steps=10, grains=1, charge="consistent",
             plasma="maxwell", mach=1.0, collisions="none", force="allpairs", rc=0.0, rs=0.0, tall=1,
             every=1),
        # the reference's small benchmark size (workloads.small_plain)
        dict(name="window_small_plain", kind="window", n=16384, steps=10, grains=1,
             charge="consistent", plasma="maxwell", mach=1.0, collisions="none", force="allpairs",
             rc=0.0, rs=0.0, tall=1, every=1),
        # a field-driven production run with the reference's per-component collisions, ragged size
        dict(name="window_field_driven", kind="window", n=50021, steps=10, grains=3, charge="oml",
             plasma="field", mach=0.5, collisions="per_dof", force="allpairs", rc=0.0, rs=0.0, tall=1,
             every=1),
        # the headline workload's size and physics (workloads.full_plain)
        dict(name="window_full_plain", kind="window", n=2**20, steps=1, grains=1,
             charge="consistent", plasma="maxwell", mach=1.0, collisions="mfp", force="allpairs",
             rc=0.0, rs=0.0, tall=1, every=1),
        # the dust chain with a 2 lambda cutoff (workloads.field_chain)
        dict(name="window_field_chain", kind="window", n=2**19, steps=3, grains=5,
             charge="consistent", plasma="field", mach=0.5, collisions="mfp", force="cutoff", rc=2.0,
             rs=1.875, tall=1, every=1),
        # the reference's cutoff benchmark: a domain taller than wide (workloads.cutoff_scaling)
        dict(name="window_cutoff_tall", kind="window", n=65536, steps=3, grains=1, charge="given",
             plasma="maxwell", mach=1.0, collisions="none", force="cutoff", rc=3.2, rs=3.0, tall=2,
             every=1),
        # a small run with a hard cutoff, ragged size
        dict(name="window_hard_cutoff", kind="window", n=20011, steps=10, grains=2,
             charge="consistent", plasma="maxwell", mach=1.5, collisions="none", force="cutoff",
             rc=2.0, rs=0.0, tall=1, every=1),
        # grains that move between windows (matthews.DustDynamics), tabulated trap
        dict(name="fork_dust_dynamics", kind="fork", n=30000, steps=10, grains=2, mach=1.0),
        # a chunk of a sweep or of the request server: members of different sizes and intervals
        dict(name="batch_sweep", kind="batch", members=6, log2_lo=14.0, log2_hi=17.0, steps=16,
             every="mixed"),
        # a whole call for a small study point
        dict(name="simulate_call", kind="simulate", n=8192, steps=100, grains=2, mach=0.8,
             charge="consistent"),
        # force of one frame, ordinary size
        dict(name="snapshot_allpairs", kind="snapshot", n=70001, force="allpairs", rc=0.0, rs=0.0),
        # force of a few thousand ions that another code owns
        dict(name="static_small", kind="static", n=3001),
    ]


def _log_int(rng, lo, hi):
    n = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    return max(2, n | 1 if rng.random() < 0.5 else n)


def draw(rng: random.Random):
    kind = rng.choice(["window", "window", "window", "window", "cutoff", "cutoff", "cutoff", "fork",
                       "batch", "simulate", "snapshot", "snapshot", "static"])
    if kind in ("window", "cutoff"):
        field = rng.random() < 0.4
        c = dict(kind="window", n=0, steps=1, grains=rng.randint(1, 5), charge=rng.choice(METHODS),
                 plasma="field" if field else "maxwell", mach=round(rng.uniform(0.2, 2.0), 3),
                 collisions=rng.choice(["per_dof", "mfp"] if field else ["none", "mfp"]),
                 force="allpairs", rc=0.0, rs=0.0, tall=1, every=1)
        if kind == "cutoff":
            c["n"] = _log_int(rng, 4096, 2**19)
            c["tall"] = rng.choice([1, 1, 2, 4])
            c["force"] = "cutoff"
            c["rc"] = round(rng.uniform(1.5, 3.2) if c["n"] < 2**17 else rng.uniform(1.5, 2.0), 3)
            c["rs"] = 0.0 if rng.random() < 0.35 else round(c["rc"] * 0.9375, 4)
        else:
            c["n"] = _log_int(rng, 1024, 600000)
            c["every"] = rng.choice([1, 1, 1, 4])
        c["steps"] = 16 if c["n"] < 40000 else (8 if c["n"] < 150000 else 4 if c["every"] == 4 else 2)
        return c
    if kind == "fork":
        return dict(kind="fork", n=_log_int(rng, 4096, 100000), steps=rng.choice([5, 10, 20]),
                    grains=rng.randint(1, 4), mach=round(rng.uniform(0.4, 1.6), 3))
    if kind == "batch":
        lo = rng.uniform(14.0, 15.5)
        return dict(kind="batch", members=rng.randint(2, 8), log2_lo=round(lo, 3),
                    log2_hi=round(lo + rng.uniform(0.5, 2.0), 3), steps=16,
                    every=rng.choice(["mixed", "one", "sixteen"]))
    if kind == "simulate":
        return dict(kind="simulate", n=_log_int(rng, 2048, 40000), steps=rng.choice([30, 60, 100, 150]),
                    grains=rng.randint(1, 4), mach=round(rng.uniform(0.2, 2.0), 3),
                    charge=rng.choice(METHODS))
    if kind == "snapshot":
        force = rng.choice(["allpairs", "cutoff"])
        rc = round(rng.uniform(1.5, 3.2), 3) if force == "cutoff" else 0.0
        return dict(kind="snapshot", n=_log_int(rng, 512, 120000), force=force, rc=rc,
                    rs=0.0 if force != "cutoff" or rng.random() < 0.3 else round(rc * 0.9375, 4))
    return dict(kind="static", n=_log_int(rng, 64, 32768))


# ------------------------------------------------------------------ parameter objects
M_AR, T_I, T_E, N_INF = workloads.M_AR, workloads.T_I, workloads.T_E, workloads.N_INF


def _plasma(case):
    if case.get("plasma") != "field":
        return od.PlasmaParametersInSIUnitsMaxwell(T_I, T_E, N_INF, case.get("mach", 1.0), M_AR)
    # field-driven as workloads.field_chain: mean free path 1 lambda at the given Mach number
    k_B, e = 1.380649e-23, 1.60217662e-19
    v_B, v_T = math.sqrt(k_B * T_E / M_AR), math.sqrt(k_B * T_I / M_AR)
    lam = math.sqrt(8.85418781762039e-12 * k_B * T_E / (e**2 * N_INF))
    v_fl = case["mach"] * v_B
    w_c = math.sqrt(v_fl**2 + 8 * v_T**2 / math.pi) / lam
    return od.PlasmaParametersInSIUnitsFieldDriven(T_I, T_E, N_INF, v_fl * M_AR * w_c / e, w_c, M_AR)


def _chain(n_grains, lam, charge, r=5e-6, gap=1.0):
    q = -1.0e-15 if charge == "given" else 0.0
    return [od.DustParticle(0.0, 0.0, (k - (n_grains - 1) / 2.0) * gap * lam, r, charge, q)
            for k in range(n_grains)]


def _engine(case, seed, rows):
    plasma = _plasma(case)
    lam = plasma.r_D_e
    sim = od.SimulationParametersInSIUnits(3 * lam, 6 * lam * case["tall"], case["n"], rows, 1e-10,
                                           plasma)
    ext = {}
    if case["collisions"] == "mfp":
        ext.update(collisions="mfp", mean_free_path=2 * lam if case["plasma"] == "maxwell" else lam)
    if case["force"] == "cutoff":
        ext.update(cutoff_distance=case["rc"] * lam, switch_distance=case["rs"] * lam)
    dist = "fieldDriven" if case["plasma"] == "field" else "Maxwellian"
    holder, _ = od.build_simulation(plasma, sim, _chain(case["grains"], lam, case["charge"]), dist,
                                    seed=seed, force_every=case["every"], **ext)
    eng = _lib.Engine(holder)
    if dist == "fieldDriven":
        eng.init_state(setup_host.field_driven_vz_table(plasma.v_fl, plasma.v_T))
    else:
        eng.init_state()
    return eng


def _snapshot_positions(n, R, H, rng):
    """Uniform in the cylinder (Debye lengths), FP32 values: a state as the device holds it."""
    r = R * np.sqrt(rng.random(n))
    th = 2 * np.pi * rng.random(n)
    z = H * (rng.random(n) - 0.5)
    return np.stack([r * np.cos(th), r * np.sin(th), z], 1).astype(np.float32).astype(np.float64)


def _snapshot_case(case, seed):
    """Plasma, simulation parameters and positions [m] of a snapshot or static case."""
    plasma = od.PlasmaParametersInSIUnitsMaxwell(T_I, T_E, N_INF, 1.0, M_AR)
    lam = plasma.r_D_e
    sim = od.SimulationParametersInSIUnits(3 * lam, 6 * lam, case["n"], 4, 1e-10, plasma)
    x = _snapshot_positions(case["n"], 3.0, 6.0, np.random.default_rng(seed))
    return plasma, sim, x * lam


# ------------------------------------------------------------------ prepare
def prepare(case, seed):
    kind = case["kind"]
    if kind == "window":
        return dict(kind=kind, eng=_engine(case, seed, SERIES_ROWS), steps=case["steps"])
    if kind == "fork":
        phi = {"E_0": [2600.0, "V/m"], "alpha": [2.4e6, "V/m^2"], "beta": [3.0e8, "V/m^3"],
               "z1": [-1.0e-3, "m"], "z7": [1.5e-3, "m"]}
        plasma = matthews.PlasmaParametersInSIUnitsMatthews(290.0, 30000.0, 1e14, 2, phi,
                                                            case["mach"], 2e6, 6.6335209e-26)
        lam = plasma.r_D_e
        sim = matthews.SimulatioParametersInSIUnits(1.25 * lam, 5 * lam, case["n"], case["steps"],
                                                    2e-10, plasma)
        grains = [matthews.DustParticle(0.0, 0.0, g.z, 4.4e-6, "consistent", -1.5e-15)
                  for g in _chain(case["grains"], lam, "consistent", gap=0.6)]
        holder = matthews.build_matthews(plasma, sim, grains, seed=seed, consider_trap=False)
        eng = _lib.Engine(holder)
        eng.init_state()
        table = matthews.fit_trap(eng, plasma, sim)
        q_s = abs(plasma.e) * sim.N_s
        xyz = np.array([[g.x, g.y, g.z] for g in grains])
        eng.set_trap_table(table, setup_host.trap_table_out_factor(
            table, sim.H, lam, plasma.eps_0, q_s, [tuple(p) for p in xyz]))
        field = matthews.grain_field(plasma, xyz[:, 2])
        return dict(kind=kind, eng=eng, steps=case["steps"], xyz=xyz, q=np.full(len(grains), -1.5e-15),
                    field=field)
    if kind == "batch":
        rng = np.random.default_rng(seed)
        sizes = np.random.default_rng(7919 * case["members"] + int(1000 * case["log2_lo"]))
        every = {"mixed": (1, 4, 8, 16), "one": (1,), "sixteen": (16,)}[case["every"]]
        batch, slots = _lib.Batch(), []
        for m in range(case["members"]):
            n = int(round(2 ** sizes.uniform(case["log2_lo"], case["log2_hi"])))
            c = dict(n=n, grains=1 + m % 4, charge="consistent", plasma="maxwell",
                     mach=float(rng.uniform(0.1, 2.0)))
            plasma = _plasma(c)
            lam = plasma.r_D_e
            sim = od.SimulationParametersInSIUnits(3 * lam, 6 * lam, n, SERIES_ROWS, 1e-10, plasma)
            ext = dict(collisions="mfp", mean_free_path=2 * lam) if m % 2 else {}
            holder, _ = od.build_simulation(plasma, sim, _chain(c["grains"], lam, "consistent"),
                                            "Maxwellian", seed=seed * 64 + m,
                                            force_every=every[m % len(every)], **ext)
            slots.append(batch.add(holder))
        return dict(kind=kind, batch=batch, slots=slots, steps=case["steps"])
    if kind == "simulate":
        plasma = od.PlasmaParametersInSIUnitsMaxwell(T_I, T_E, N_INF, case["mach"], M_AR)
        lam = plasma.r_D_e
        sim = od.SimulationParametersInSIUnits(3 * lam, 6 * lam, case["n"], case["steps"], 1e-10,
                                               plasma)
        return dict(kind=kind, plasma=plasma, sim=sim, seed=seed,
                    grains=_chain(case["grains"], lam, case["charge"]))
    plasma, sim, pos = _snapshot_case(case, seed)
    lam = plasma.r_D_e
    if kind == "snapshot":
        ext = {}
        if case["force"] == "cutoff":
            ext = dict(cutoff_distance=case["rc"] * lam, switch_distance=case["rs"] * lam)
        holder, _ = od.build_simulation(plasma, sim, _chain(1, lam, "consistent"), "Maxwellian",
                                        seed=seed, trap=np.zeros(15), **ext)
        return dict(kind=kind, eng=_lib.Engine(holder), pos=pos)
    q_s = abs(plasma.e) * sim.N_s
    return dict(kind=kind, lib=_lib.load(), n=case["n"], lam=lam, r_0=sim.r_0,
                kqq=q_s * q_s / (4.0 * np.pi * plasma.eps_0),
                pos=torch.tensor(pos, dtype=torch.float64, device="cuda"),
                force=torch.empty((case["n"], 3), dtype=torch.float64, device="cuda"))


# ------------------------------------------------------------------ run
def _f32(a):
    return a.astype(np.float32)


def _results(eng, first, count):
    s = eng.series(first, count)
    pos, vel = eng.get_state()
    return dict(q=s["q"], dust=s["dust"], orbit=_f32(s["orbit"]), collect=_f32(s["collect"]),
                pos=_f32(pos), vel=_f32(vel))


def run(state):
    kind = state["kind"]
    if kind == "window":
        eng, k = state["eng"], state["steps"]
        if eng.step_index + k > eng.n_steps:
            eng.begin_window()
        first = eng.step_index
        eng.step(k)
        return _results(eng, first, k)
    if kind == "fork":
        eng, x = state["eng"], state["xyz"]
        eng.begin_window()
        eng.step(state["steps"])
        eng.set_grains(x[:, 0], x[:, 1], x[:, 2], state["q"], state["field"])
        return _results(eng, 0, state["steps"])
    if kind == "batch":
        batch, k = state["batch"], state["steps"]
        members = [batch.member(s) for s in state["slots"]]
        for m in members:
            if m.step_index + k > m.n_steps:
                m.begin_window()
        batch.step(k)
        return [_results(m, m.step_index - k, k) for m in members]
    if kind == "simulate":
        sim = od.OpenDust(state["plasma"], state["sim"], od.OutputParameters(), state["grains"],
                          "Maxwellian")
        q, forces = sim.simulate("0", seed=state["seed"], quiet=True)
        return dict(q=q, dust=forces["dust"], orbit=_f32(forces["orbit"]),
                    collect=_f32(forces["collect"]))
    if kind == "snapshot":
        return _f32(state["eng"].force_snapshot(state["pos"]))
    st = state["lib"].od_ion_forces_static(
        ctypes.c_void_p(state["pos"].data_ptr()), state["n"], state["lam"], state["r_0"],
        state["kqq"], ctypes.c_void_p(state["force"].data_ptr()),
        ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
    _lib.check(st, None)
    return state["force"].float()


# ------------------------------------------------------------------ work
def _pairs(n, force, rc, R, H):
    """Unordered pairs of n uniform ions that interact; a cutoff's share from sampled pairs."""
    pairs = n * (n - 1) / 2.0
    if force != "cutoff":
        return pairs
    rng = np.random.default_rng(1)
    a, b = _snapshot_positions(200000, R, H, rng), _snapshot_positions(200000, R, H, rng)
    return pairs * float(np.mean(np.sum((a - b) ** 2, 1) < rc * rc))


def work(case):
    # 31 flops per unordered pair (the screened term, and its sum on both ions); an ion's state
    # (position, velocity, force: 48 bytes) read and written once a step and 48 bytes of FP64
    # position and velocity handed to the caller
    kind = case["kind"]
    if kind == "batch":
        sizes = np.random.default_rng(7919 * case["members"] + int(1000 * case["log2_lo"]))
        every = {"mixed": (1, 4, 8, 16), "one": (1,), "sixteen": (16,)}[case["every"]]
        flops = nbytes = 0.0
        for m in range(case["members"]):
            n = int(round(2 ** sizes.uniform(case["log2_lo"], case["log2_hi"])))
            k = every[m % len(every)]
            flops += 31.0 * n * (n - 1) / 2 * (case["steps"] // k)
            nbytes += n * (96.0 * case["steps"] + 48)
        return dict(bytes=nbytes, flops=flops)
    n = case["n"]
    if kind in ("snapshot", "static"):
        return dict(bytes=48.0 * n, flops=31.0 * _pairs(n, case.get("force"), case.get("rc"), 3.0, 6.0))
    steps = case["steps"]
    p = _pairs(n, case.get("force"), case.get("rc"), 3.0, 6.0 * case.get("tall", 1))
    return dict(bytes=n * (96.0 * steps + 48), flops=31.0 * p * max(1, steps // case.get("every", 1)))


# ------------------------------------------------------------------ exact
def exact(case, seed):
    """Forces of the snapshot and static cases in 64 bits. Whole runs have no such value here:
    their ions collide and re-enter by random draws."""
    if case["kind"] not in ("snapshot", "static"):
        return None
    plasma, sim, pos = _snapshot_case(case, seed)
    lam, rho = plasma.r_D_e, sim.r_0 / plasma.r_D_e
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    x = torch.tensor(pos, dtype=torch.float64, device=dev) / lam
    n = x.shape[0]
    cut = case.get("force") == "cutoff"
    rc, rs = case.get("rc", 0.0), case.get("rs", 0.0)
    out = torch.empty_like(x)
    step = max(1, min(n, 2**25 // n))
    for i in range(0, n, step):
        d = x[i:i + step, None, :] - x[None, :, :]
        r = torch.sqrt((d * d).sum(2))
        own = r == 0
        r = torch.where(own, torch.ones_like(r), r)
        s = 1.0 / (r + rho)
        u = torch.exp(-r) * s
        f = u * (1.0 + s)
        if cut:
            # OpenMM's switching function on the energy u between rs and rc
            if 0.0 < rs < rc:
                t = ((r - rs) / (rc - rs)).clamp(0.0, 1.0)
                f = f * (1 - t) ** 3 * (1 + 3 * t + 6 * t * t) + u * 30 * (t * (1 - t)) ** 2 / (rc - rs)
            f = torch.where(r < rc, f, torch.zeros_like(f))
        f = torch.where(own, torch.zeros_like(f), f / r)
        out[i:i + step] = (f[:, :, None] * d).sum(1)
    q_s = abs(plasma.e) * sim.N_s
    return out.cpu().numpy() * (q_s * q_s / (4.0 * np.pi * plasma.eps_0) / lam**2)
