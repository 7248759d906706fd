"""What this framework is timed on: one pass of each case is the work a
user's program has it do, through the public entry points.

`listed()` names the cases, `draw()` gives more of the same ranges,
`prepare()` makes what a program has in hand before the call, `run()` is one
pass, `work()` the bytes and operations a pass cannot do without, and
`exact()` the same result in 64 bits from plain torch.

Scenes are the package's own benchmark configurations (sand column, NACC
snowball, dam breach, mixed batch) and demo scenes in size, spacing and
material, in a loaded state: lattices with jitter, a falling, shearing body
and a compressed deformation gradient, so that constraints, contacts, return
maps and the water's density solve all have work. Bodies are aligned with
the grid's cells (two lattice planes per cell, as the dam breach's columns
are in x and y).
"""
import importlib
import math

import numpy as np
import torch

xp = importlib.import_module("xpbi-webgpu_gb300")
_abi = importlib.import_module("xpbi-webgpu_gb300._abi")
net = importlib.import_module("xpbi-webgpu_gb300.net")
train_warm = importlib.import_module("xpbi-webgpu_gb300.train_warm")
S = xp.scenes

JITTER = 0.27  # of the spacing: about one solid particle in a hundred is in contact
WATER_JITTER = 0.1
WATER_SPACING = 1.0035  # of the spacing: near the density solve's rest state (a lattice at 1 is 1% too dense)


def listed():
    return [
        # the smallest benchmark config, one substep per call: latency and launches
        {"name": "column_16k", "kind": "step", "body": "column", "nx": 20, "ny": 40, "nz": 20, "iterations": 10},
        # the browser demo's frame on its plasticine ball: uniforms, a few substeps, positions to the host
        {"name": "demo_frame_8k", "kind": "frame", "body": "plasticine", "radius": 0.16, "iterations": 6,
         "substeps": 4},
        # the demo's water over sand: few iterations, a PBF pass after each
        {"name": "demo_dam_27k", "kind": "step", "body": "demo_dam", "nx": 9, "ny": 17, "nz": 47, "iterations": 3,
         "pbf": -1},
        # a checkpointed / logged substep of a small viscoplastic body: the whole state to the host
        {"name": "record_goo_9k", "kind": "record", "body": "goo", "radius": 0.171, "iterations": 3},
        # an all-solid body of middle size with the most iterations
        {"name": "snowball_113k", "kind": "step", "body": "snowball", "radius": 0.3, "iterations": 20},
        # a middling dam breach of odd extents, with the reference's PBF pass after every iteration
        {"name": "dam_100k_interleaved", "kind": "step", "body": "dam", "nx": 61, "ny": 53, "nz": 31,
         "iterations": 7, "pbf": -1},
        # the one-million-particle dam breach
        {"name": "dam_1m", "kind": "step", "body": "dam", "nx": 125, "ny": 80, "nz": 100, "iterations": 15, "pbf": 4},
        # the headline mix: four of them in one handle, plain solve ...
        {"name": "dam_mix_4m", "kind": "step", "body": "dam", "nx": 125, "ny": 80, "nz": 100, "iterations": 15,
         "pbf": 4, "scenes": 4},
        # ... and the learned solve (network warm start, active set, early stop)
        {"name": "dam_mix_4m_learned", "kind": "learned", "body": "dam", "nx": 125, "ny": 80, "nz": 100,
         "iterations": 15, "pbf": 4, "scenes": 4},
        # many uneven scenes with every plasticity model in one handle
        {"name": "batch_256", "kind": "step", "body": "batch", "scenes": 256, "lo": 2000, "hi": 60000,
         "iterations": 20},
        # the warm-start network's training: Adam steps on mini-batches from host rows
        {"name": "train_8192x24", "kind": "train", "rows": 65536, "batch": 8192, "steps": 24},
        # the cell sort alone, on the caller's device buffers
        {"name": "sort_250k", "kind": "sort", "n": 250007},
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    body = rng.choice(["column", "column", "snowball", "snowball", "dam", "dam", "dam", "batch", "batch", "goo",
                       "plasticine", "demo_dam", "train", "sort"])
    if body == "column":
        n = _log(rng, 2000, 120000)
        nx, nz = rng.randint(11, 40), rng.randint(11, 40)
        return {"kind": "step", "body": body, "nx": nx, "ny": max(5, min(46, int(n / (nx * nz)))), "nz": nz,
                "iterations": rng.randint(5, 20)}
    if body == "snowball":
        return {"kind": "step", "body": body, "radius": round(_log(rng, 0.06, 0.34), 4),
                "iterations": rng.randint(5, 20)}
    if body == "goo":
        return {"kind": "record", "body": body, "radius": round(rng.uniform(0.1, 0.25), 4),
                "iterations": rng.randint(2, 6)}
    if body == "plasticine":
        return {"kind": "frame", "body": body, "radius": round(rng.uniform(0.08, 0.3), 4),
                "iterations": rng.randint(2, 6), "substeps": rng.randint(2, 5)}
    if body == "demo_dam":
        return {"kind": "step", "body": body, "nx": rng.randint(5, 10), "ny": rng.randint(7, 24),
                "nz": rng.randint(9, 47), "iterations": rng.randint(2, 5), "pbf": -1}
    if body == "batch":
        return {"kind": "step", "body": body, "scenes": int(_log(rng, 3, 200)), "lo": 2000,
                "hi": int(_log(rng, 8000, 60000)), "iterations": rng.randint(10, 20)}
    if body == "train":
        b = int(_log(rng, 700, 16384))
        return {"kind": "train", "rows": 4 * b, "batch": b, "steps": rng.randint(8, 32)}
    if body == "sort":
        return {"kind": "sort", "n": int(_log(rng, 1000, 262144))}
    nx, ny, nz = rng.randint(30, 125), rng.randint(25, 80), max(9, int(_log(rng, 9, 100)))
    kind = rng.choice(["step", "step", "step", "learned"])
    return {"kind": kind, "body": "dam", "nx": nx, "ny": ny, "nz": nz, "iterations": rng.randint(12 if kind == "learned" else 6, 15),
            "pbf": 4 if kind == "learned" else rng.choice([-1, 2, 4]), "scenes": rng.choice([1, 1, 2])}


# ---------------------------------------------------------------- scenes
def _aligned_sphere(rng, pos, mid, st, radius, h, state0, corner):
    """A sphere whose lattice planes lie half a spacing off the grid's cells."""
    c = [x + 0.5 * h + math.ceil(radius / h) * h for x in corner]
    r = math.ceil(radius / h) * h
    tmp = []
    S.sample_sphere(rng, tmp, [], [], c, r, h, 0, 0.0, state0)
    p = tmp[0][((tmp[0] - np.array(c)) ** 2).sum(1) <= radius ** 2]
    pos.append(p + (rng.random(p.shape) - 0.5) * JITTER * h)
    mid.append(np.zeros(len(p), np.uint32))
    st.append(np.full(len(p), state0))


def _scene(h, dmin, dmax, materials, rng, build, dt, gravity, **solver):
    s = S.base(h)
    pos, mid, st = [], [], []
    build(pos, mid, st)
    p = np.concatenate(pos).astype(np.float32)
    s.update(domainMin=list(dmin), domainMax=list(dmax), positions=p, matIds=np.concatenate(mid),
             states=np.concatenate(st).astype(np.float32), materials=materials,
             hasWater=any(m["kind"] == S.WATER for m in materials),
             colorSeeds=(rng.random(len(p)) * 0.49).astype(np.float32), gravity=[0.0, gravity, 0.0], dt=dt, **solver)
    return s


def _box(rng, pos, mid, st, corner, n, h, mat, state0=0.0, jitter=JITTER):
    hi = [corner[k] + n[k] * h for k in range(3)]
    S.sample_box(rng, pos, mid, st, corner, hi, h, mat, jitter, state0)


def _water(rng, pos, mid, st, corner, n, h, mat):
    """Water near the rest state of its density solve: the lattice stretched about its middle."""
    tmp = []
    _box(rng, tmp, mid, st, corner, n, h, mat, 0.0, WATER_JITTER)
    middle = np.array(corner) + np.array(n) * (h / 2)
    pos.append(middle + (tmp[0] - middle) * WATER_SPACING)


def _bounds(p, h):
    """A box around a body, four cells of padding on five sides, the floor close below; aligned with the cells."""
    lo = [float(np.floor(p[:, k].min() / (2 * h)) * 2 * h - 8 * h) for k in range(3)]
    lo[1] += 8 * h
    return lo, [float(np.ceil(p[:, k].max() / (2 * h)) * 2 * h + 8 * h) for k in range(3)]


def _batch_scene(rng, sizes, case):
    """One scene of the mixed batch: sizes, materials and iteration counts as the 256-scene config draws them. The
    sizes come from `sizes`, which is the same for every seed of a case."""
    h, values, rng = 0.01, rng, sizes
    target = math.exp(rng.uniform(math.log(case["lo"]), math.log(case["hi"])))
    E = math.exp(rng.uniform(math.log(5e4), math.log(5e5)))
    kind = int(rng.choice([S.DP, S.NACC, S.VM, S.HB, S.SNOW]))
    m = {S.DP: dict(density=1000.0, p0=S.dp_alpha(float(rng.uniform(25, 40))), p1=0.0),
         S.NACC: dict(density=400.0, p0=-0.04, p1=0.5, p2=3.0, p3=1.85),
         S.VM: dict(density=1000.0, p0=math.exp(rng.uniform(math.log(1e3), math.log(1e4)))),
         S.HB: dict(density=1000.0, p0=float(rng.uniform(50, 500)), p1=float(rng.uniform(0.3, 1.0)),
                    p2=float(rng.uniform(1, 50))),
         S.SNOW: dict(density=400.0, p0=2.5e-2, p1=7.5e-3, p2=10.0)}[kind]
    m.update(kind=kind, E=E, nu=0.3, color=[0.8, 0.8, 0.8], boundFriction=0.4)
    state0 = {S.NACC: -0.04, S.SNOW: 1.0}.get(kind, 0.0)
    sphere = rng.random() < 0.5
    side = max(2, round((target / 2) ** (1 / 3)))

    def build(pos, mid, st):
        if sphere:
            _aligned_sphere(values, pos, mid, st, h * (3 * target / (4 * math.pi)) ** (1 / 3), h, state0, [0.1] * 3)
        else:
            _box(values, pos, mid, st, [0.1] * 3, (side, max(2, round(target / side ** 2)), side), h, 0, state0)
    s = _scene(h, [0.0] * 3, [1.0] * 3, [m], values, build, 1e-4, -9.81,
               iterations=int(rng.integers(max(1, case["iterations"] // 2), case["iterations"] + 1)))
    s["domainMin"], s["domainMax"] = _bounds(s["positions"], h)
    return s


def _scenes(case, seed):
    """The case's scenes, each with a loaded state (velocities, F, plastic state)."""
    rng, sizes = np.random.default_rng(seed), np.random.default_rng(7)
    body, it = case["body"], case["iterations"]
    out = []
    for _ in range(case.get("scenes", 1)):
        if body == "column":  # Drucker-Prager sand standing on the floor
            h, n = 0.01, (case["nx"], case["ny"], case["nz"])
            m = dict(kind=S.DP, E=1e5, nu=0.3, density=1600.0, p0=S.dp_alpha(30), p1=0.0, color=[0.85, 0.63, 0.28],
                     boundFriction=0.5)
            s = _scene(h, [0.0] * 3, [1.0, 0.5, 1.0], [m], rng,
                       lambda p, q, t: _box(rng, p, q, t, [0.3, 0.0, 0.3], n, h, 0), 2e-4, -9.81, iterations=it)
        elif body == "snowball":  # NACC sphere thrown at a wall
            h = 0.01
            m = dict(kind=S.NACC, E=1.4e5, nu=0.3, density=400.0, p0=-0.04, p1=0.5, p2=3.0, p3=1.85,
                     color=[0.93, 0.95, 0.98], boundFriction=0.35)
            s = _scene(h, [0.0] * 3, [1.0] * 3, [m], rng,
                       lambda p, q, t: _aligned_sphere(rng, p, q, t, case["radius"], h, -0.04, [0.04, 0.16, 0.16]),
                       1e-4, -9.81, iterations=it)
        elif body == "goo":  # Herschel-Bulkley sphere of the demo
            h = 0.013
            s = _scene(h, [0.0] * 3, [1.0] * 3, [S.GOO(1.0)], rng,
                       lambda p, q, t: _aligned_sphere(rng, p, q, t, case["radius"], h, 0.0, [0.338] * 3), 1 / 1080,
                       -9.8, iterations=it)
        elif body == "plasticine":  # von Mises sphere of the demo
            h = 0.013
            s = _scene(h, [0.0] * 3, [1.0] * 3, [S.PLASTICINE(80)], rng,
                       lambda p, q, t: _aligned_sphere(rng, p, q, t, case["radius"], h, 0.0, [0.182] * 3),
                       0.4 / 480, -9.8, iterations=it)
        elif body == "demo_dam":  # the demo's water over a sand dam
            h, (nx, ny, nz) = 0.019, (case["nx"], case["ny"], case["nz"])

            def build(p, q, t):
                _box(rng, p, q, t, [0.418, 0.0, 0.038], (nx, ny, nz), h, 0)
                _water(rng, p, q, t, [0.038, 0.0, 0.038], (nx + 8, ny + 8, nz), h, 1)
            s = _scene(h, [0.0] * 3, [1.0] * 3, [S.SAND(30, 0.004), S.WATER_MAT()], rng, build, 1.25e-3, -9.8,
                       iterations=it, pbfIterations=None)
        elif body == "dam":  # water (60%) beside a Drucker-Prager dam, 8 mm
            h, (nx, ny, nz) = 0.008, (case["nx"], case["ny"], case["nz"])
            wet = (3 * nx) // 5
            sand = dict(kind=S.DP, E=2e5, nu=0.3, density=1600.0, p0=S.dp_alpha(35), p1=0.0,
                        color=[0.85, 0.63, 0.28], boundFriction=0.5)
            water = dict(kind=S.WATER, E=100, nu=0.3, density=1000.0, color=[0.25, 0.55, 0.95], boundFriction=0.0)

            def build(p, q, t):
                _water(rng, p, q, t, [0.016, 0.0, 0.096], (wet, ny, nz), h, 1)
                _box(rng, p, q, t, [0.016 + 2 * h * ((wet + 1) // 2), 0.0, 0.096], (nx - wet, ny, nz), h, 0)
            s = _scene(h, [0.0] * 3, [2.0, 1.0, 1.0], [sand, water], rng, build, 1e-4, -9.81, iterations=it,
                       pbfIterations=None if case["pbf"] < 0 else case["pbf"])
        else:
            s = _batch_scene(rng, sizes, case)
        _load(s, rng, thrown={"snowball": -3.0, "dam": 10.0, "plasticine": 0.0}.get(body, 2.0))
        out.append(s)
    return out


def _load(s, rng, thrown):
    """A moving, shearing body under load: smooth velocities with a little noise, F compressed by a few permille."""
    p = s["positions"].astype(np.float64)
    n, h = len(p), s["h"]
    k = 2 * math.pi / (40 * h)
    wave = 0.1 * np.stack([np.sin(k * p[:, 1]), np.sin(k * p[:, 2]), np.sin(k * p[:, 0])], 1)
    v = wave + rng.standard_normal((n, 3)) * 0.01
    v[:, 1] -= 0.1
    v[:, 0] += thrown
    s["velocities"] = v.astype(np.float32)
    depth = (p[:, 1].max() - p[:, 1]) / max(p[:, 1].max() - p[:, 1].min(), h)
    F = rng.standard_normal((n, 3, 3)) * 1e-3 + np.eye(3) * (1 - 0.002 - 0.003 * depth)[:, None, None]
    s["F"] = F.astype(np.float32)  # [particle, column, row]


def _F12(F):
    out = np.zeros((len(F), 12), np.float32)
    out.reshape(-1, 3, 4)[:, :, :3] = F
    return out


_streams = []


def _stream():
    """The stream a program runs its simulations on, one after the other."""
    if not _streams:
        _streams.append(torch.cuda.Stream())
    return _streams[0].cuda_stream


class _DeviceArray:
    """A borrowed device pointer as an array other libraries can view; a view of it keeps the handle that owns the
    memory."""

    def __init__(self, owner, ptr, shape, typestr="<f4"):
        self.owner = owner
        self.__cuda_array_interface__ = {"shape": shape, "typestr": typestr, "data": (ptr, False), "version": 3}


# ---------------------------------------------------------------- prepare / run
def prepare(case, seed):
    kind = case["kind"]
    if kind == "train":
        return _train_inputs(case, seed)
    if kind == "sort":
        return _sort_inputs(case, seed)
    scenes = _scenes(case, seed)
    sim = xp.Simulation(scenes if len(scenes) > 1 else scenes[0])
    sim.set_stream(_stream())
    params = [xp.params_for(s) for s in scenes]
    wet = any(s["hasWater"] for s in scenes)
    for k, s in enumerate(scenes):
        sim.write_params(params[k], scene=k)
        sim.set_schedule(k, s["iterations"], s["hasWater"])
        sim.write_state(k, F=_F12(s["F"]))
    st = {"case": case, "sim": sim, "params": params, "wet": wet, "iterations": case["iterations"]}
    if kind == "learned":
        # tolerances as the plain solve reaches them on this scene, the active set and the cap of the benchmark
        sim.set_network(train_warm.load_weights())
        sim.set_active_set(0.25)
        sim.set_max_iterations(30)
        sim.set_solver(sim.NETWORK, 2.2e-4, False, False, contact_rel_tol=2.4e-2)
    if kind in ("step", "learned"):
        p, v, _ = sim.device_ptrs()
        for k, ptr in (("pos", p), ("vel", v)):
            st[k] = torch.as_tensor(_DeviceArray(sim, ptr, (sim.N, 4)), device="cuda")
            st[k].owner = sim
    if kind == "frame":
        st["host"] = np.empty((sim.N, 4), np.float32)
    return st


def run(st):
    case = st["case"]
    kind = case["kind"]
    if kind in ("step", "learned"):
        st["sim"].step(1, -1, st["wet"])
        return {"pos": st["pos"], "vel": st["vel"]}
    if kind == "frame":
        sim = st["sim"]
        sim.write_params(st["params"][0])
        sim.step(case["substeps"], st["iterations"], st["wet"])
        return {"pos": sim.read_pos(out=st["host"])}
    if kind == "record":
        st["sim"].encode_substep(st["iterations"], st["wet"])
        return st["sim"].read_state()
    if kind == "train":
        p, loss = net.train(st["X"], st["T"], st["p"], steps=case["steps"], batch=case["batch"], lr=2e-3)
        return {"params": p, "loss": loss}
    if kind == "sort":
        _abi.check(_abi.lib().xpbi_sort_cells_noalloc(st["pos"].data_ptr(), case["n"], st["origin"], st["cs"],
                                                      st["dims"], st["start"].data_ptr(), st["idx"].data_ptr(),
                                                      torch.cuda.current_stream().cuda_stream))
        return {"start": st["start"], "idx": st["idx"]}
    raise ValueError(kind)


def _train_inputs(case, seed):
    rng = np.random.default_rng(seed)
    X = rng.standard_normal((case["rows"], 16)).astype(np.float32)
    T = np.tanh(X @ rng.standard_normal(16).astype(np.float32) * 0.5) + 0.3 * X[:, 0] * X[:, 1]
    w = [rng.standard_normal(64 * 16) * math.sqrt(2 / 16), rng.standard_normal(64) * 0.1,
         rng.standard_normal(64 * 64) * math.sqrt(2 / 64), rng.standard_normal(64) * 0.1,
         rng.standard_normal(64 * 64) * math.sqrt(2 / 64), rng.standard_normal(64) * 0.1,
         rng.standard_normal(64) * math.sqrt(1 / 64), rng.standard_normal(1) * 0.1]
    return {"case": case, "X": X, "T": T.astype(np.float32), "p": np.concatenate(w).astype(np.float32)}


def _sort_inputs(case, seed):
    """Particles of a block at eight per cell, in the order of an earlier substep's cells (slightly disturbed)."""
    import ctypes as C
    n, h = case["n"], 0.01
    g = torch.Generator(device="cuda").manual_seed(seed)
    side = max(2, round(n ** (1 / 3)))
    i = torch.arange(n, device="cuda")
    q = torch.stack([i % side, (i // side) % side, i // side ** 2], 1) + torch.rand(n, 3, generator=g, device="cuda") * 1.6
    pos = torch.zeros(n, 4, device="cuda")
    pos[:, :3] = q * h + 4 * h
    dims = [side // 2 + 6, side // 2 + 6, (n // side ** 2) // 2 + 7]
    return {"case": case, "pos": pos.contiguous(), "origin": (C.c_float * 3)(0.0, 0.0, 0.0), "cs": 2 * h,
            "dims": (C.c_int32 * 3)(*dims), "cells": dims[0] * dims[1] * dims[2],
            "start": torch.zeros(dims[0] * dims[1] * dims[2] + 1, dtype=torch.int32, device="cuda"),
            "idx": torch.zeros(n, dtype=torch.int32, device="cuda")}


def work(case):
    """Bytes: the state (position, velocity, F, plastic state: 72 B per particle) read once and written once per
    substep, plus what goes to the host. Operations: the pair sums and per-particle tails the method states, at 33
    neighbours (a support of two spacings)."""
    kind = case["kind"]
    if kind == "train":
        macs = 64 * 16 + 2 * 64 * 64 + 64
        return {"bytes": case["rows"] * 68 + 2 * 4 * 9473, "flops": 6 * macs * case["batch"] * case["steps"]}
    if kind == "sort":
        return {"bytes": case["n"] * 20, "flops": case["n"] * 12}
    solid, water = _counts(case)
    n = solid + water
    it, pbf = case["iterations"], case.get("pbf", 0)
    it = it * 0.75 if case["body"] == "batch" else it
    passes = it if pbf < 0 else min(pbf, it)
    per = 33 * 45 * it * 2 + 900 * it + 33 * 90 + 600
    f = solid * per + water * (33 * 45 * 2 * passes + 33 * 20) + n * 200
    subs = case.get("substeps", 1)
    host = 16 * n if kind == "frame" else 132 * n if kind == "record" else 0
    return {"bytes": 144 * n * subs + host, "flops": f * subs}


def _counts(case):
    body = case["body"]
    if body == "column":
        return case["nx"] * case["ny"] * case["nz"], 0
    if body in ("snowball", "goo", "plasticine"):
        return round(4 / 3 * math.pi * (case["radius"] / (0.01 if body == "snowball" else 0.013)) ** 3), 0
    if body == "batch":
        return round(case["scenes"] * (case["hi"] - case["lo"]) / math.log(case["hi"] / case["lo"])), 0
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    if body == "demo_dam":
        return nx * ny * nz, (nx + 8) * (ny + 8) * nz
    wet = (3 * nx) // 5
    k = case.get("scenes", 1)
    return k * (nx - wet) * ny * nz, k * wet * ny * nz


# ---------------------------------------------------------------- exact
def exact(case, seed):
    kind = case["kind"]
    if kind in ("step", "record"):
        out = _Exact(_scenes(case, seed)).substep()
        if kind == "step":
            return {"pos": out["pos"], "vel": out["vel"]}
        return {"pos": out["pos"], "vel": out["vel"], "F": out["F"], "L": out["L"], "aux": None, "sortedIdx": None,
                "cellTab": None}
    if kind == "train":
        return _exact_train(case, seed)
    return None  # several substeps, an early stop by residuals, or integers


def _exact_train(case, seed):
    st = _train_inputs(case, seed)
    X, T = (torch.tensor(st[k], dtype=torch.float64, device="cuda") for k in ("X", "T"))
    p = torch.tensor(st["p"], dtype=torch.float64, device="cuda", requires_grad=True)
    m, v = torch.zeros_like(p), torch.zeros_like(p)
    cut = np.cumsum([0, 1024, 64, 4096, 64, 4096, 64, 64, 1])
    loss, off, b = [], 0, case["batch"]
    for t in range(case["steps"]):
        if off + b > case["rows"]:
            off = 0
        w = [p[cut[k]:cut[k + 1]] for k in range(8)]
        a = X[off:off + b]
        for k, i in ((0, 16), (2, 64), (4, 64)):
            a = torch.nn.functional.silu(a @ w[k].view(64, i).T + w[k + 1])
        e = ((a @ w[6] + w[7] - T[off:off + b]) ** 2).mean()
        g, = torch.autograd.grad(e, p)
        loss.append(e.detach())
        with torch.no_grad():
            m = 0.9 * m + 0.1 * g
            v = 0.999 * v + 0.001 * g * g
            p -= 2e-3 * (m / (1 - 0.9 ** (t + 1))) / (torch.sqrt(v / (1 - 0.999 ** (t + 1))) + 1e-8)
        off += b
    return {"params": p.detach(), "loss": torch.stack(loss)}


def _f32(x):
    return float(np.float32(x))


class _Exact:
    """One substep of several scenes in 64 bits, from the method's own equations (plain torch, no part of the
    package's kernels): cell sort, Bonet-Lok correction, XPBI iterations with contact and walls, PBF, XSPH, the
    plastic update. The cell of a particle is formed in 32 bits, since it decides the order of the results."""

    def __init__(self, scenes):
        d = dict(dtype=torch.float64, device="cuda")
        self.sc = scenes
        s0, p0 = scenes[0], xp.params_for(scenes[0])
        self.h, self.dt = _f32(s0["h"]), _f32(p0["dt"])
        self.H = _f32(2 * s0["h"])
        self.V0 = _f32(s0["h"] ** 3)
        self.g = torch.tensor([_f32(x) for x in s0["gravity"]], **d)
        self.omega, self.gamma, self.comega = _f32(p0["omega"]), _f32(p0["kDamp"]), _f32(p0["contactOmega"])
        self.xsph, self.eps, self.scorr = _f32(p0["xsphC"]), _f32(p0["pbfEps"]), _f32(p0["sCorrK"])
        self.alpha = 1 / self.V0 / self.dt ** 2
        self.sigW = 21 / (16 * 3.14159265 * self.h ** 3)
        cat = lambda f, t=torch.float32: torch.cat([torch.as_tensor(f(s), device="cuda").to(t) for s in scenes])
        self.x32 = cat(lambda s: s["positions"])
        self.w = cat(lambda s: s["matIds"].astype(np.float32) + s["colorSeeds"])
        self.v = cat(lambda s: s["velocities"], torch.float64)
        self.F = cat(lambda s: s["F"], torch.float64).transpose(1, 2).contiguous()  # rows, columns
        self.state = cat(lambda s: s["states"], torch.float64)
        self.sid = torch.cat([torch.full((len(s["positions"]),), k, dtype=torch.int64, device="cuda")
                              for k, s in enumerate(scenes)])
        self.mat = cat(lambda s: s["matIds"].astype(np.int64), torch.int64) + 8 * self.sid
        mats = [dict(s["materials"][m]) if m < len(s["materials"]) else None for s in scenes for m in range(8)]

        def col(f):
            return torch.tensor([_f32(f(m)) if m else 0.0 for m in mats], **d)
        self.kind = torch.tensor([m["kind"] if m else 0 for m in mats], device="cuda")
        self.mu = col(lambda m: m["E"] / (2 * (1 + m["nu"])))
        self.lam = col(lambda m: m["E"] * m["nu"] / ((1 + m["nu"]) * (1 - 2 * m["nu"])))
        self.rho = col(lambda m: m["density"])
        self.mass = col(lambda m: m["density"] * s0["h"] ** 3)
        self.fric = col(lambda m: 0.4 if m.get("boundFriction") is None else m["boundFriction"])
        self.par = torch.stack([col(lambda m, k=k: m.get("p%d" % k) or 0.0) for k in range(4)], 1)
        self.lo = torch.tensor([[_f32(x) for x in s["domainMin"]] for s in scenes], **d)
        self.hi = torch.tensor([[_f32(x) for x in s["domainMax"]] for s in scenes], **d)
        self.iters = torch.tensor([s["iterations"] for s in scenes], device="cuda")
        self.pbf = [0 if not s["hasWater"] else s["iterations"] if s.get("pbfIterations") is None
                    else min(s["iterations"], s["pbfIterations"]) for s in scenes]

    # -- cells and neighbours
    def _sort(self):
        cs = 2 * self.sc[0]["h"]
        org, dims, base, total = [], [], [], 0
        for s in self.sc:
            org.append([_f32(a - 2 * cs) for a in s["domainMin"]])
            n = [math.ceil((s["domainMax"][k] - s["domainMin"][k]) / cs) + 4 for k in range(3)]
            dims.append(n)
            base.append(total)
            total += n[0] * n[1] * n[2]
        o = torch.tensor(org, dtype=torch.float32, device="cuda")[self.sid]
        self.dims = torch.tensor(dims, device="cuda")
        self.base = torch.tensor(base, device="cuda")
        c = torch.floor((self.x32 - o) / np.float32(cs)).clamp(min=0)
        c = torch.minimum(c.long(), self.dims[self.sid] - 1)
        nd = self.dims[self.sid]
        key = self.base[self.sid] + c[:, 0] + c[:, 1] * nd[:, 0] + c[:, 2] * nd[:, 0] * nd[:, 1]
        back = torch.arange(len(key) - 1, -1, -1, device="cuda")
        order = back[torch.sort(key[back], stable=True)[1]]  # by cell, within a cell by descending index
        for k in ("x32", "w", "v", "F", "state", "sid", "mat"):
            setattr(self, k, getattr(self, k)[order])
        self.x = self.x32.double()
        self.cell = c[order]
        self.count = torch.bincount(key, minlength=total)
        self.start = torch.cumsum(self.count, 0) - self.count
        self.n = len(order)

    def _neighbours(self, x, who):
        """Padded neighbour lists of the particles `who`: those of the 27 cells around each within the support at
        the positions x, itself as padding."""
        m = int(self.count.max())
        lists, most = [], 1
        off = torch.tensor([[a, b, c] for c in (-1, 0, 1) for b in (-1, 0, 1) for a in (-1, 0, 1)], device="cuda")
        for i in who.split(1 << 17):
            c = self.cell[i][:, None, :] + off
            nd = self.dims[self.sid[i]][:, None, :]
            ok = ((c >= 0) & (c < nd)).all(2)
            k = (self.base[self.sid[i]][:, None] + c[..., 0] + c[..., 1] * nd[..., 0]
                 + c[..., 2] * nd[..., 0] * nd[..., 1]).clamp(0, len(self.start) - 1)
            j = self.start[k][..., None] + torch.arange(m, device="cuda")
            ok = ok[..., None] & (torch.arange(m, device="cuda") < self.count[k][..., None])
            j = torch.where(ok, j, i[:, None, None]).flatten(1)
            near = ((x[j] - x[i][:, None]) ** 2).sum(2) < self.H ** 2
            near &= j != i[:, None]
            num = near.sum(1)
            most = max(most, int(num.max()) if len(num) else 1)
            row, at = near.nonzero(as_tuple=True)
            lists.append((i, j[row, at].int(), row, num))
        out = torch.empty(len(who), most, dtype=torch.int32, device="cuda")
        done = 0
        for i, j, row, num in lists:
            o = out[done:done + len(i)]
            o.copy_(i[:, None].expand(-1, most))
            o[row, torch.arange(len(row), device="cuda") - (torch.cumsum(num, 0) - num)[row]] = j
            done += len(i)
        return out

    @staticmethod
    def _each(who, nb, f):
        """f over pieces of (particles, their lists), its results joined."""
        got = [f(i, j.long()) for i, j in zip(who.split(1 << 18), nb.split(1 << 18))]
        return [torch.cat(t) for t in zip(*got)]

    def _grad(self, dx):
        """Gradient of the Wendland C2 kernel."""
        t = (1 - dx.norm(dim=-1, keepdim=True) / (2 * self.h)).clamp(min=0)
        return dx * (-5 * self.sigW / self.h ** 2 * t ** 3)

    @staticmethod
    def _svd(F):
        """V and singular values of 3x3 F by Jacobi rotations of F^T F."""
        A = F.transpose(1, 2) @ F
        a = {(i, j): A[:, i, j].clone() for i in range(3) for j in range(i, 3)}
        V = [[torch.full_like(a[0, 0], float(i == j)) for j in range(3)] for i in range(3)]
        for _ in range(7):
            for p, q in ((0, 1), (0, 2), (1, 2)):
                r = 3 - p - q
                apq = a[p, q]
                tau = (a[q, q] - a[p, p]) / (2 * torch.where(apq == 0, torch.ones_like(apq), apq))
                t = torch.where(tau >= 0, 1.0, -1.0) / (tau.abs() + torch.sqrt(1 + tau * tau))
                t = torch.where(apq == 0, torch.zeros_like(t), t)
                c = 1 / torch.sqrt(1 + t * t)
                s = t * c
                a[p, p], a[q, q] = a[p, p] - t * apq, a[q, q] + t * apq
                a[p, q] = torch.zeros_like(apq)
                kp, kq = (min(p, r), max(p, r)), (min(q, r), max(q, r))
                a[kp], a[kq] = c * a[kp] - s * a[kq], s * a[kp] + c * a[kq]
                for k in range(3):
                    V[k][p], V[k][q] = c * V[k][p] - s * V[k][q], s * V[k][p] + c * V[k][q]
        sig = torch.stack([a[i, i].clamp(min=0).sqrt() for i in range(3)], 1)
        return torch.stack([torch.stack(r, 1) for r in V], 1), sig

    # -- material models
    def _map(self, sig, mat, state, mu, lam):
        kind, par = self.kind[mat], self.par[mat]
        out, st = sig.clone(), state.clone()
        safe = sig.clamp(1e-3, 1e3)
        for k in set(kind.tolist()) if len(kind) < 100 else set(torch.unique(kind).tolist()):
            i = (kind == k).nonzero()[:, 0]
            s, p, m, l = safe[i], par[i], mu[i], lam[i]
            if k == S.DP:
                coh = p[:, 1:2]
                e = torch.log(s) - coh
                tr = e.sum(1, keepdim=True)
                dev = e - tr / 3
                dn = dev.norm(dim=1, keepdim=True)
                dg = dn + p[:, :1] * ((3 * l + 2 * m) / (2 * m))[:, None] * tr
                en = torch.exp(e - dg / dn.clamp(min=1e-300) * dev + coh)
                r = torch.where(dg <= 0, sig[i], en)
                out[i] = torch.where((dn < 1e-9) | (tr > 0), torch.exp(coh).expand_as(r), r)
            elif k == S.VM:
                e = torch.log(s)
                dev = e - e.mean(1, keepdim=True)
                dn = dev.norm(dim=1, keepdim=True)
                dg = dn - (p[:, 0] / (2 * m))[:, None]
                out[i] = torch.where((dg <= 0) | (dn < 1e-9), sig[i], torch.exp(e - dg / dn.clamp(min=1e-300) * dev))
            elif k == S.HB:
                out[i] = self._herschel_bulkley(sig[i], s, p, m)
            elif k == S.NACC:
                out[i], st[i] = self._nacc(sig[i], s, p, m, l, state[i])
            elif k == S.SNOW:
                new = torch.minimum(torch.maximum(sig[i], 1 - p[:, :1]), 1 + p[:, 1:2])
                out[i] = new
                st[i] = (state[i] * sig[i].prod(1) / new.prod(1).clamp(min=1e-6)).clamp(0.2, 2.0)
        return out, st

    def _herschel_bulkley(self, sig, s, p, mu):
        J = s.prod(1)
        b = s * s * (J ** (-2 / 3))[:, None]
        trb = b.sum(1)
        dev = b - trb[:, None] / 3
        pre = mu * dev.norm(dim=1)
        sy = math.sqrt(2 / 3) * p[:, 0]
        mt = trb / 3 * mu
        hexp, eta = p[:, 1], p[:, 2]
        lin = ((hexp - 1).abs() < 1e-3) | (eta < 1e-9)
        new = pre - (pre - sy) / (1 + eta / (2 * mt * self.dt))
        ih = 1 / hexp
        lo, hi = sy.clone(), pre.clone()
        for _ in range(18):
            mid = 0.5 * (lo + hi)
            g = eta ** ih * (mid - pre) + 2 * mt * self.dt * (mid - sy).clamp(min=0) ** ih
            hi, lo = torch.where(g > 0, mid, hi), torch.where(g > 0, lo, mid)
        new = torch.where(lin, new, 0.5 * (lo + hi))
        bn = (dev * (new / pre.clamp(min=1e-300))[:, None] + trb[:, None] / 3).clamp(min=1e-6)
        bn = bn * (bn.prod(1) ** (-1 / 3))[:, None]
        return torch.where(((pre <= sy) | (pre < 1e-12))[:, None], sig, bn.sqrt() * (J ** (1 / 3))[:, None])

    def _nacc(self, sig, s, p, mu, lam, state):
        beta, xi, M = p[:, 1], p[:, 2], p[:, 3]
        kap = 2 / 3 * mu + lam
        J = s.prod(1)
        b2 = s * s
        trb = b2.sum(1)
        sh = (mu * J ** (-2 / 3))[:, None] * (b2 - trb[:, None] / 3)
        sn = sh.norm(dim=1)
        q = math.sqrt(1.5) * sn
        pr = -0.5 * kap * (J * J - 1)
        a = state.clamp(-0.25, 0.4)
        p0 = kap * (0.00001 + torch.sinh((xi * (-a).clamp(min=0)).clamp(max=4.0)))
        b = 1 + 2 * beta
        J1 = (-2 * p0 / kap + 1).clamp(min=1e-6).sqrt()
        J2 = (2 * beta * p0 / kap + 1).clamp(min=1e-6).sqrt()
        c1, c2 = pr > p0, pr < -beta * p0
        y = b * q * q + M * M * (pr + beta * p0) * (pr - p0)
        c3 = ~c1 & ~c2 & (y > 1e-4) & (sn > 1e-9)
        # hardening toward the intersection with the yield surface
        pc = (1 - beta) * p0 * 0.5
        ln = torch.sqrt((pc - pr) ** 2 + q * q)
        Dp, Dq = (pc - pr) / ln.clamp(min=1e-300), -q / ln.clamp(min=1e-300)
        A = M * M * Dp * Dp + b * Dq * Dq
        B = M * M * Dp * (2 * pc - p0 + beta * p0)
        Cq = M * M * (pc + beta * p0) * (pc - p0)
        disc = B * B - 4 * A * Cq
        r = disc.clamp(min=0).sqrt()
        A2 = 2 * torch.where(A == 0, torch.ones_like(A), A)
        px1, px2 = pc + (-B + r) / A2 * Dp, pc + (-B - r) / A2 * Dp
        px = torch.where((pr - pc) * (px2 - pc) > 0, px2, px1)
        Jx2 = -2 * px / kap + 1
        hard = c3 & (p0 > 1e-4) & (pr < p0 - 1e-4) & (pr > -beta * p0 + 1e-4) & (ln > 1e-9) & (disc > 0) \
            & (A.abs() > 1e-12) & (Jx2 > 1e-8)
        Jx = Jx2.clamp(min=1e-300).sqrt()
        an = torch.where(hard & (Jx > 1e-4), a + torch.log(J / Jx), a)
        an = torch.where(c1, a + torch.log(J / J1), torch.where(c2, a + torch.log(J / J2), an))
        qn = M * ((-(pr + beta * p0) * (pr - p0)).clamp(min=0) / b).sqrt()
        bn = (J ** (2 / 3) / mu * (qn / math.sqrt(1.5)) / sn.clamp(min=1e-300))[:, None] * sh + trb[:, None] / 3
        out = torch.where(c3[:, None], bn.clamp(min=1e-6).sqrt(), sig)
        out = torch.where(c1[:, None], (J1 ** (1 / 3))[:, None].expand_as(out), out)
        return torch.where(c2[:, None], (J2 ** (1 / 3))[:, None].expand_as(out), out), an

    def _hard(self, mat, state):
        """Lame parameters, snow's hardened by its state."""
        mu, lam = self.mu[mat], self.lam[mat]
        s = torch.where(self.kind[mat] == S.SNOW, torch.exp((self.par[mat][:, 2] * (1 - state)).clamp(max=5.0)),
                        torch.ones_like(mu))
        return mu * s, lam * s

    # -- the substep
    def _walls(self, x, v):
        xq = x + self.dt * v
        lo, hi = self.lo[self.sid], self.hi[self.sid]
        fr = self.fric[self.mat]
        for k in range(3):
            out = (xq[:, k] < lo[:, k]) | (xq[:, k] > hi[:, k])
            bound = torch.where(xq[:, k] < lo[:, k], lo[:, k], hi[:, k])
            vn = (bound - x[:, k]) / self.dt
            vt = v.clone()
            vt[:, k] = 0
            tl = vt.norm(dim=1)
            drop = torch.minimum(fr * (vn - v[:, k]).abs(), tl)
            nv = torch.where((tl > 1e-9)[:, None], v - vt / tl.clamp(min=1e-300)[:, None] * drop[:, None], v)
            nv[:, k] = vn
            v = torch.where(out[:, None], nv, v)
            xq = torch.where(out[:, None], x + self.dt * v, xq)
        return v

    def substep(self):
        self._sort()
        dt, x = self.dt, self.x
        self.Vn = self.V0 * torch.linalg.det(self.F).clamp(0.1, 10.0)
        v = self.v + self.g * dt
        water = self.kind[self.mat] == S.WATER
        sol = (~water).nonzero()[:, 0]
        everyone = torch.arange(self.n, device="cuda")
        nb = self._neighbours(x, everyone)
        nbs = nb[sol]  # of the solids
        nbs_solid = torch.where(water[nbs.long()], sol[:, None].int(), nbs)
        mass = self.mass[self.mat]
        mS, FS, stS, matS = mass[sol], self.F[sol], self.state[sol], self.mat[sol]
        mu, lam = self._hard(matS, stS)

        def correction(i, j):
            r = x[j] - x[i][:, None]
            A = torch.einsum("nka,nkb,nk->nab", self._grad(-r), r, self.Vn[j])
            V, s = self._svd(A)
            d = torch.where(s > 0.2, 1 / (s * s).clamp(min=1e-300), torch.zeros_like(s))
            return (V * d[:, None, :]) @ V.transpose(1, 2) @ A.transpose(1, 2),
        # only the solids' enters the substep; the water's is part of the whole state
        L_all, = self._each(everyone, nb, correction) if self.n < 50000 else (None,)
        L = L_all[sol] if L_all is not None else self._each(sol, nbs, correction)[0]

        def sums(i, j):
            gj = self._grad(x[i][:, None] - x[j])
            Vb = self.Vn[j]
            return (gj * Vb[..., None]).sum(1), torch.einsum("nka,nkb,nk->nab", gj, gj, Vb * Vb / mass[j])
        sg, P = self._each(sol, nbs_solid, sums)
        sv = (L @ sg[..., None])[..., 0]
        Q = L @ P @ L.transpose(1, 2)

        def velocity_gradient(i, j):
            gj = self._grad(x[i][:, None] - x[j])
            return torch.einsum("nka,nkb,nk->nab", v[j] - v[i][:, None], gj, self.Vn[j]),
        mult = torch.zeros(len(sol), dtype=torch.float64, device="cuda")
        eye = torch.eye(3, dtype=torch.float64, device="cuda")
        slot = torch.zeros(self.n, dtype=torch.int64, device="cuda")
        slot[sol] = torch.arange(len(sol), device="cuda")
        for k in range(int(self.iters.max())):
            on = self.iters[self.sid] > k
            G = self._each(sol, nbs_solid, velocity_gradient)[0] @ L.transpose(1, 2)
            Ft = (eye + dt * G) @ FS
            V, s0 = self._svd(Ft)
            sig, _ = self._map(s0, matS, stS, mu, lam)
            e = torch.log(sig.clamp(1e-3, 1e3))
            tr = e.sum(1)
            C = torch.sqrt((2 * (mu * (e * e).sum(1) + 0.5 * lam * tr * tr)).clamp(min=0))
            act = (C >= 1e-7) & on[sol]
            dpsi = (2 * mu[:, None] * e + (lam * tr)[:, None]) / sig.clamp(1e-3, 1e3)
            d = dpsi / C.clamp(min=1e-300)[:, None] / s0.clamp(min=1e-300)
            M = Ft @ (V * d[:, None, :]) @ V.transpose(1, 2) @ FS.transpose(1, 2)
            gs = -(M @ sv[..., None])[..., 0]
            den = ((M.transpose(1, 2) @ M) * Q).sum((1, 2)) + (gs * gs).sum(1) / mS
            cdot = (M * G).sum((1, 2))
            dl = self.omega * (-C - self.alpha * mult - self.gamma * dt * cdot) / ((1 + self.gamma) * den + self.alpha)
            dl = torch.where(act, dl, torch.zeros_like(dl))
            mult = mult + dl
            R = (M @ L) * dl[:, None, None]
            xc = x + dt * v

            def impulses(i, j):
                dx = x[j] - x[i][:, None]
                dv = torch.einsum("nkab,nkb->na", R[slot[j]], self._grad(dx)) * self.Vn[i][:, None]
                dc = xc[i][:, None] - xc[j]
                dist = dc.norm(dim=2)
                wgt = mass[j] / (mass[i][:, None] + mass[j]) * (0.75 * self.h - dist).clamp(min=0)
                wgt = torch.where((dist > 1e-9) & (j != i[:, None]), wgt / dist.clamp(min=1e-300),
                                  torch.zeros_like(dist))
                return dv, (dc * wgt[..., None]).sum(1)
            dv, corr = self._each(sol, nbs_solid, impulses)
            dv = (dv + gs * dl[:, None]) / (mS * dt)[:, None]
            size = dv.norm(dim=1)
            cap = 0.2 * self.H / dt
            dv = torch.where((size > cap)[:, None], dv * (cap / size.clamp(min=1e-300))[:, None], dv)
            new = v.clone()
            new[sol] += dv + corr * (self.comega / dt)
            v = torch.where(on[:, None], self._walls(x, new), v)
            if any(k < p for p in self.pbf):
                v = self._pbf(v, water)
        v = self._xsph(v, water, nb)
        G = self._each(sol, nbs_solid, velocity_gradient)[0] @ L.transpose(1, 2)
        Ft = (eye + dt * G) @ FS
        V, s0 = self._svd(Ft)
        sig, st = self._map(s0, matS, stS, mu, lam)
        F = self.F.clone()
        F[sol] = Ft @ (V * (sig.clamp(1e-3, 1e3) / s0.clamp(min=1e-300))[:, None, :]) @ V.transpose(1, 2)
        size = v.norm(dim=1)
        cap = 0.45 * self.H / dt
        v = torch.where((size > cap)[:, None], v * (cap / size.clamp(min=1e-300))[:, None], v)
        xn = torch.minimum(torch.maximum(x + dt * v, self.lo[self.sid]), self.hi[self.sid])

        def planes(A):
            out = torch.zeros(len(A), 3, 4, dtype=torch.float64, device="cuda")
            out[:, :, :3] = A.transpose(1, 2)
            return out.reshape(-1, 12)
        return {"pos": torch.cat([xn, self.w.double()[:, None]], 1), "vel": torch.cat([v, self.Vn[:, None]], 1),
                "F": planes(F), "L": planes(L_all) if L_all is not None else None}

    def _pbf(self, v, water):
        dt, H = self.dt, self.H
        xc = x = self.x + dt * v
        k6 = 315 / (64 * 3.14159265 * H ** 9)
        ks = -45 / (3.14159265 * H ** 6)
        wat = water.nonzero()[:, 0]
        mass, rho0 = self.mass[self.mat], self.rho[self.mat]
        everyone = torch.arange(self.n, device="cuda")
        nb = self._neighbours(xc, everyone)

        def spiky(dx):
            r = dx.norm(dim=-1, keepdim=True)
            return torch.where(r < 1e-9, torch.zeros_like(dx), dx * (ks * (H - r).clamp(min=0) ** 2
                                                                     / r.clamp(min=1e-300)))

        def density(i, j):
            dx = xc[i][:, None] - xc[j]
            w6 = k6 * (H * H - (dx * dx).sum(2)).clamp(min=0) ** 3
            mb = torch.where(j != i[:, None], mass[j], torch.zeros_like(w6))
            r = mass[i] * k6 * H ** 6 + (mb * w6).sum(1)
            gr = spiky(dx) * (mb / rho0[i][:, None])[..., None]
            s = gr.sum(1)
            return -(r / rho0[i] - 1).clamp(min=0) / ((gr * gr).sum((1, 2)) + (s * s).sum(1) + self.eps),
        lw, = self._each(wat, nb[wat], density)
        lam = torch.zeros(self.n, dtype=torch.float64, device="cuda")
        lam[wat] = lw
        w0 = k6 * (H * H - (0.2 * H) ** 2) ** 3

        def shift(i, j):
            dx = xc[i][:, None] - xc[j]
            wj, wi = water[j], water[i][:, None]
            use = (wj | wi) & (j != i[:, None])
            rel = k6 * (H * H - (dx * dx).sum(2)).clamp(min=0) ** 3 / max(w0, 1e-12)
            mpd = torch.where(wj, mass[j] / rho0[j], (mass / rho0)[i][:, None])
            f = torch.where(use, (lam[i][:, None] + lam[j] - self.scorr * rel ** 4) * mpd, torch.zeros_like(rel))
            return (spiky(dx) * f[..., None]).sum(1),
        dp, = self._each(everyone, nb, shift)
        del x
        return v + dp * (torch.where(water, 1.0, 0.5) / dt)[:, None]

    def _xsph(self, v, water, nb):
        def mix(i, j):
            q = (self.x[i][:, None] - self.x[j]).norm(dim=2) / self.h
            t = (1 - 0.5 * q).clamp(min=0)
            wgt = torch.where(water[j] == water[i][:, None], self.sigW * t ** 4 * (2 * q + 1) * self.Vn[j],
                              torch.zeros_like(q))
            return ((v[j] - v[i][:, None]) * wgt[..., None]).sum(1),
        acc, = self._each(torch.arange(self.n, device="cuda"), nb, mix)
        return v + (torch.where(water, 10 * self.xsph, self.xsph)[:, None]) * acc
