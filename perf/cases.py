"""Performance cases: the work a user of the solver has it do.

A case is one of five kinds of work, each through the public Python entry
points, with the default tile shapes unless the caller it stands for sets
them:

* ``sim``     a whole simulation on a handle the program keeps: zero the
              state, set the source, step, read the surface records and the
              final displacement back into pinned host buffers;
* ``request`` the same with a new crystal loaded into the handle first, as
              the serving loop does when a pooled simulation gets a request;
* ``plugin``  ``Solver.init`` + ``Solver.run`` of the plugin, as the
              application's run button does: everything is created anew;
* ``batch``   many uneven crystals stepped together, joined, stepped in
              chunks of 60 and read back as the serving loop does;
* ``energy``  the energy of a state in mid-run, the error metric of a run.

Crystals are those of the benchmark configurations: a silicon-like host with
a lattice of voids and tungsten cylinders, drawn from the seed.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from phonomena_gb300.batch import Batch
from phonomena_gb300.device import DeviceSimulation
from phonomena_gb300.model import Grid, Material
from phonomena_gb300.solver_gb300 import Solver

FIELDS = ("ux", "uy", "uz")
# bytes a node cannot do without per step (displacement, velocity and Kahan
# term read and written in FP32, or u_old, u read and u_new written in FP64,
# and the material id) and the operations of the scheme
STEP_BYTES = {"f32k": 73, "f64": 73, "f64v": 145}
STEP_FLOPS = {"f32k": 105, "f64": 105, "f64v": 105}
ENERGY_FLOPS = 60


def _sim(name, cells, precision, steps, **kw):
    case = {"name": name, "kind": "sim", "nx": cells[0], "ny": cells[1], "nz": cells[2], "precision": precision,
            "steps": steps, "pitch": 16, "surface_mode": "corrected", "bc": "absorbing", "source_mode": "line",
            "graded": False, "record_every": 10}
    case.update(kw)
    return case


def listed():
    return [
        # the smallest runs: a mesh of a few thousand nodes while a model is set
        # up, the plugin's default arithmetic and the reference's surface row
        _sim("tiny_f64", (24, 20, 12), "f64", 100, pitch=8, surface_mode="reference"),
        # the reference's own speed-test mesh (60 x 60 x 20 cells, 1000 steps)
        # from the application, inclusions and all
        {"name": "plugin_f64", "kind": "plugin", "nx": 60, "ny": 60, "nz": 20, "precision": "f64", "steps": 1000,
         "pitch": 12, "surface_mode": "reference", "record_every": 10},
        # the first benchmark crystal (40 x 40 x 20 cells, 500 steps) in the
        # fast arithmetic: parameter sweeps over small crystals
        _sim("small_f32k", (40, 40, 20), "f32k", 500, pitch=8),
        # a mesh refined towards its middle, as the application builds around
        # an inclusion: odd extents, dozens of distinct spacings
        _sim("graded_f64", (149, 130, 46), "f64", 120, pitch=12, graded=True),
        # the headline crystal, shortened from 2000 steps
        _sim("crystal_f32k", (256, 256, 128), "f32k", 360),
        # the same crystal in the reference's arithmetic
        _sim("crystal_f64", (256, 256, 128), "f64", 60),
        # a large crystal (68 million nodes): the range of the precision runs
        _sim("large_f32k", (512, 512, 256), "f32k", 96),
        # the FP64 form of the fast scheme, on odd extents, with the rigid
        # walls and the plane source
        _sim("odd_f64v", (193, 161, 97), "f64v", 120, bc="rigid", source_mode="wall"),
        # a request of the serving loop on a pooled simulation
        {**_sim("request_f32k", (160, 128, 64), "f32k", 300, pitch=8), "kind": "request"},
        # the serving mix: crystals of {64..192}^2 x {32..96} cells side by
        # side on worker streams, with the serving loop's tile shape
        {"name": "serve_batch_f32k", "kind": "batch", "count": 24, "low": 64, "high": 192, "low_z": 32, "high_z": 96,
         "mix": 4, "precision": "f32k", "steps": 180, "streams": 64, "tile_j": 16, "record_every": 10},
        # the default batch (persistent launches) over smaller crystals
        {"name": "batch_f32k", "kind": "batch", "count": 12, "low": 48, "high": 128, "low_z": 24, "high_z": 64,
         "mix": 9, "precision": "f32k", "steps": 180, "streams": 0, "tile_j": 8, "record_every": 10},
        # the energy of the headline crystal's state
        {"name": "energy_f32k", "kind": "energy", "nx": 256, "ny": 256, "nz": 128, "precision": "f32k", "pitch": 16},
    ]


def _between(rng, lo, hi):
    """An integer of lo..hi, spread over the logarithm."""
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["sim"] * 6 + ["request", "plugin", "batch", "batch", "energy", "energy"])
    precision = rng.choice(["f64", "f64", "f32k", "f32k", "f32k", "f64v"])
    pitch = rng.choice([8, 12, 16])
    every = rng.choice([5, 10])
    if kind == "plugin":
        return {"kind": "plugin", "nx": _between(rng, 24, 96), "ny": _between(rng, 24, 96), "nz": _between(rng, 10, 32),
                "precision": rng.choice(["f64", "f32k"]), "steps": rng.randint(100, 1000), "pitch": pitch,
                "surface_mode": "corrected", "record_every": every}
    if kind == "batch":
        streams = rng.choice([0, 64])
        low, low_z = rng.randint(40, 80), rng.randint(20, 40)
        return {"kind": "batch", "count": rng.randint(6, 24), "low": low, "high": rng.randint(low, 192), "low_z": low_z,
                "high_z": rng.randint(low_z, 96), "mix": rng.randrange(1 << 20), "precision": "f32k",
                "steps": rng.randint(24, 180), "streams": streams, "tile_j": 16 if streams else rng.choice([8, 16]),
                "record_every": every}
    if kind == "energy":
        while True:
            nx, ny, nz = _between(rng, 20, 320), _between(rng, 20, 320), _between(rng, 12, 160)
            if nx * ny * nz <= 256 * 256 * 128:
                return {"kind": "energy", "nx": nx, "ny": ny, "nz": nz, "precision": rng.choice(["f32k", "f64"]),
                        "pitch": pitch}
    # whole simulations: a mesh of 10^3.5 to 10^7.8 nodes, and as many steps
    # as keep the run below the largest listed one of its arithmetic
    top = {"f32k": 68e6 if kind == "sim" else 4e6, "f64": 8.5e6, "f64v": 8.5e6}[precision]
    budget = {"f32k": 3e9, "f64": 4e8, "f64v": 4e8}[precision]
    while True:
        nx, ny, nz = _between(rng, 16, 640), _between(rng, 16, 640), _between(rng, 10, 288)
        if 4000 <= nx * ny * nz <= top:
            break
    most = int(min(600, budget / (nx * ny * nz)))
    case = _sim("", (nx, ny, nz), precision, rng.randint(max(24, most // 2), max(30, most)), pitch=pitch,
                bc=rng.choice(["absorbing", "absorbing", "rigid"]), source_mode=rng.choice(["line", "line", "wall"]),
                graded=precision == "f64" and nx * ny * nz < 2e6 and rng.random() < 0.3, record_every=every)
    del case["name"]
    return {**case, "kind": kind}


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
# stiffness rows C00..C22, C33, C44, C55 (Pa) and density: host, void, tungsten
def _isotropic(lam, mu, rho):
    d = lam + 2 * mu
    return [d, lam, lam, lam, d, lam, lam, lam, d, mu, mu, mu, rho]


TABLE = np.array([_isotropic(64e9, 80e9, 2330.0), [0.0] * 12 + [2330.0], _isotropic(200e9, 160e9, 19300.0)])
DX = 1e-5  # 10 um cells


def _spacing(case):
    """Full and staggered spacings per axis; a graded mesh is finer by up to
    four in its middle, in steps of 15 percent."""
    out = {}
    for ax in "xyz":
        n = case["n" + ax]
        fd = np.full(n, DX)
        if case.get("graded") and ax != "z":
            away = np.abs(np.arange(n) - n // 2) // 4
            fd = DX * np.minimum(1.0, 0.25 * 1.15 ** away)
        out["fd" + ax] = fd
        out["sd" + ax] = (fd[1:] + fd[:-1]) / 2
    return out


def _ids(nodes, pitch, rng):
    """Lattice of vertical cylinders through the top ten cells, radius
    U[0.2, 0.4] pitches, a quarter of them tungsten, the rest void; the cells
    whose cylinder would reach an absorbing wall stay solid."""
    nx, ny, nz = nodes
    px, py = -(-(nx - 1) // pitch), -(-(ny - 1) // pitch)
    radius = rng.uniform(0.2, 0.4, (px, py)) * pitch
    kind = np.where(rng.uniform(size=(px, py)) < 0.25, 2, 1)
    cx, cy = (np.arange(px) + 0.5) * pitch, (np.arange(py) + 0.5) * pitch
    wall = (cx[:, None] + radius > nx - 2) | (cy[None] + radius > ny - 2) | (cy[None] - radius < 1)
    kind[wall] = 0
    ix, iy = np.minimum(np.arange(nx) // pitch, px - 1), np.minimum(np.arange(ny) // pitch, py - 1)
    d2 = ((np.arange(nx) - cx[ix]) ** 2)[:, None] + ((np.arange(ny) - cy[iy]) ** 2)[None]
    plane = np.where(d2 < radius[ix][:, iy] ** 2, kind[ix][:, iy], 0).astype(np.uint8)
    ids = np.zeros(nodes, np.uint8)
    ids[:, :, :11] = plane[:, :, None]
    return ids


def _crystal(case, seed):
    """Spacings, ids, table, time step (half the Courant limit of the fastest
    material) and source samples of one crystal."""
    rng = np.random.default_rng(seed)
    nodes = (case["nx"] + 1, case["ny"] + 1, case["nz"] + 1)
    sp = _spacing(case)
    dt = 0.5 * min(sp["fd" + a].min() for a in "xyz") / math.sqrt(TABLE[0, 0] / TABLE[0, 12])
    freq = rng.uniform(20e6, 60e6)
    src = np.sin(2 * np.pi * freq * dt * np.arange(case["steps"])) if "steps" in case else None
    return {"spacing": sp, "ids": _ids(nodes, case["pitch"], rng), "table": TABLE, "dt": dt, "source": src,
            "surface_mode": case.get("surface_mode", "corrected"), "bc": case.get("bc", "absorbing"),
            "source_mode": case.get("source_mode", "line")}


# the application's materials: gallium arsenide with gold inclusions (10 GPa)
GAAS = {"p": 5307, "c": [[11.88, 5.87, 5.38, 0, 0, 0], [5.87, 11.88, 5.38, 0, 0, 0], [5.87, 5.38, 11.88, 0, 0, 0],
                         [0, 0, 0, 5.94, 0, 0], [0, 0, 0, 0, 5.94, 0], [0, 0, 0, 0, 0, 5.94]]}
GOLD = {"p": 19300, "c": [[19.25, 16.3, 16.3, 0, 0, 0], [16.3, 19.25, 16.3, 0, 0, 0], [16.3, 16.3, 19.25, 0, 0, 0],
                          [0, 0, 0, 4.24, 0, 0], [0, 0, 0, 0, 4.24, 0], [0, 0, 0, 0, 0, 4.24]]}


def _inclusions(case, seed):
    """Cylinders (x, y, r) on a lattice, clear of the walls, to half the depth."""
    rng = np.random.default_rng(seed)
    a = case["pitch"]
    return [(x, y, float(np.float32(rng.uniform(0.2, 0.4) * a))) for x in range(a, case["nx"] - a // 2, a)
            for y in range(a, case["ny"] - a // 2, a)], 200.0 * rng.uniform(0.7, 1.4)


def _instances(case, seed):
    """(case, seed) of each crystal of a batch: sizes and step counts belong
    to the case, the crystals to the seed."""
    mix = np.random.default_rng(case["mix"])
    out = []
    for q in range(case["count"]):
        nx, ny = (int(v) for v in mix.integers(case["low"], case["high"] + 1, 2))
        nz = int(mix.integers(case["low_z"], case["high_z"] + 1))
        out.append(({"nx": nx, "ny": ny, "nz": nz, "pitch": int(mix.choice([8, 12, 16])),
                     "steps": int(mix.integers(case["steps"] // 2, case["steps"] + 1))}, 1000 * seed + q))
    return out


def _state_fields(case, seed):
    """Displacement and velocity (or the displacement one step earlier) of a
    travelling wave packet with a weak incoherent part, on the GPU."""
    gen = torch.Generator("cuda").manual_seed(seed)
    dt = 0.5 * DX / math.sqrt(TABLE[0, 0] / TABLE[0, 12])
    real = torch.float32 if case["precision"] == "f32k" else torch.float64
    out = {}
    for c, f in enumerate(FIELDS):
        shape = [case["n" + a] + (q != c) for q, a in enumerate("xyz")]
        x, y, z = (torch.arange(n, device="cuda", dtype=torch.float64) for n in shape)
        k = 0.2 + 0.6 * torch.rand(3, generator=gen, device="cuda", dtype=torch.float64)
        wave = torch.exp(-((x - 0.4 * shape[0]) / (0.3 * shape[0])) ** 2)[:, None, None] * torch.exp(-z / 12)[None, None]
        phase = (k[0] * x)[:, None, None] + (k[1] * y)[None, :, None] + (k[2] * z)[None, None]
        noise = 1e-3 * torch.rand(shape, generator=gen, device="cuda", dtype=torch.float64)
        out[f] = (wave * torch.sin(phase) + noise).to(real)
        omega = 2 * math.pi * 42e6
        if case["precision"] == "f64":
            out[f + "_old"] = wave * torch.sin(phase - omega * dt) + noise
        else:
            out["v" + f[1]] = (omega * wave * torch.cos(phase)).to(real)
    return out, dt


# ---------------------------------------------------------------------------
# a pass
# ---------------------------------------------------------------------------
def _handle(p, case, **kw):
    sim = DeviceSimulation(p["spacing"], p["ids"], p["table"], p["dt"], precision=case["precision"],
                           surface_mode=p["surface_mode"], bc=p["bc"], source_mode=p["source_mode"],
                           max_steps=len(p["source"]), record_every=case["record_every"], **kw)
    sim.set_source(p["source"])
    return sim


def _pinned(shape, dtype):
    return torch.empty(tuple(shape), dtype=dtype, pin_memory=True).numpy()


def _buffers(ids, case, steps, fields=FIELDS):
    """Pinned host buffers for the results of one simulation."""
    real = torch.float32 if case["precision"] == "f32k" else torch.float64
    nx, ny, nz = ids.shape
    out = {"surface": _pinned((steps // case["record_every"], nx, ny), real)}
    for c, f in enumerate(FIELDS):
        if f in fields:
            out[f] = _pinned((nx - (c == 0), ny - (c == 1), nz - (c == 2)), real)
    return out


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("sim", "request"):
        p = _crystal(case, seed)
        return {"kind": kind, "sim": _handle(p, case), "inputs": p, "out": _buffers(p["ids"], case, case["steps"])}
    if kind == "plugin":
        g, m = Grid(), Material()
        g.init(case["nx"], case["ny"], case["nz"])
        cyl, f = _inclusions(case, seed)
        for x, y, r in cyl:
            g.addInclusion(x, y, r, case["nz"] // 2)
        m.init(grid=g, properties={"GaAs": GAAS, "Au": GOLD})
        m.setPrimary("GaAs")
        m.setSecondary("Au")
        return {"kind": kind, "grid": g, "material": m, "steps": case["steps"],
                "cfg": {"precision": case["precision"], "surface_mode": case["surface_mode"], "write_mode": "off",
                        "record_every": case["record_every"], "wave": "sin", "wave_args": {"f": f}}}
    if kind == "batch":
        parts = [_crystal(c, s) for c, s in _instances(case, seed)]
        sims = [_handle(p, case, tile_j=case["tile_j"], x_segment=32) for p in parts]
        return {"kind": kind, "batch": Batch(case["count"], precision=case["precision"], tile_j=case["tile_j"],
                                             streams=case["streams"]),
                "sims": sims, "steps": [len(p["source"]) for p in parts],
                "out": [_buffers(p["ids"], case, len(p["source"]), ("uz",)) for p in parts]}
    fields, dt = _state_fields(case, seed)
    p = _crystal(case, seed)
    sim = DeviceSimulation(p["spacing"], p["ids"], p["table"], dt, precision=case["precision"],
                           surface_mode="corrected")
    for f, v in fields.items():
        sim.upload(f, v.cpu().numpy())
    return {"kind": kind, "sim": sim}


def run(state):
    kind = state["kind"]
    if kind == "energy":
        kinetic, strain = state["sim"].energy()
        return {"kinetic": kinetic, "strain": strain}
    if kind == "plugin":
        s = Solver()
        s.cfg.update(state["cfg"])
        s.init(state["grid"], state["material"], state["steps"])
        s.run()
        s.release()
        return {"surface": s.surface, "ux": s.g.ux, "uy": s.g.uy, "uz": s.g.uz}
    if kind == "batch":
        b, slots = state["batch"], []
        for sim, n in zip(state["sims"], state["steps"]):
            sim.reset()
            slots.append(b.add(sim, n))
        left = max(state["steps"])
        while left > 0:
            b.step(min(60, left))
            left -= 60
        b.sync()
        for slot, sim, out in zip(slots, state["sims"], state["out"]):
            b.remove(slot)
            sim.read_surface(out=out["surface"])
            sim.download("uz", out=out["uz"])
        return state["out"]
    sim, p, out = state["sim"], state["inputs"], state["out"]
    if kind == "request":
        sim.set_materials(p["ids"], p["table"])
    sim.reset()
    sim.set_source(p["source"])
    sim.step(len(p["source"]))
    sim.sync()
    sim.read_surface(out=out["surface"])
    for f in FIELDS:
        sim.download(f, out=out[f])
    return out


def work(case):
    """A step reads and writes the state and reads the ids; the results go
    out once."""
    def one(c, fields):
        n = (c["nx"] + 1) * (c["ny"] + 1) * (c["nz"] + 1)
        size = 4 if case["precision"] == "f32k" else 8
        out = (c["steps"] // case["record_every"]) * (c["nx"] + 1) * (c["ny"] + 1) + fields * n
        return n * c["steps"] * STEP_BYTES[case["precision"]] + out * size, n * c["steps"] * STEP_FLOPS[case["precision"]]

    if case["kind"] == "energy":
        n = (case["nx"] + 1) * (case["ny"] + 1) * (case["nz"] + 1)
        return {"bytes": n * (6 * (4 if case["precision"] == "f32k" else 8) + 1), "flops": n * ENERGY_FLOPS}
    parts = [c for c, _ in _instances(case, 0)] if case["kind"] == "batch" else [case]
    done = [one(c, 1 if case["kind"] == "batch" else 3) for c in parts]
    return {"bytes": sum(b for b, _ in done), "flops": sum(f for _, f in done)}


# ---------------------------------------------------------------------------
# the same in 64 bits, with plain torch operations
# ---------------------------------------------------------------------------
def _leapfrog(p, every):
    """u_new = 2u - u_old + dt^2/rho div T(u) on the staggered grid, with the
    traction-free z = 0 row and the absorbing (or rigid) walls: the surface
    records and the final displacement."""
    dev = torch.device("cuda" if torch.cuda.is_available() else "cpu")
    ids = torch.from_numpy(p["ids"]).to(dev).long()
    nx, ny, nz = ids.shape
    tab = torch.from_numpy(np.ascontiguousarray(p["table"])).to(dev)
    dt, rows = p["dt"], [tab[:, q].contiguous() for q in range(13)]
    sp = {k: torch.from_numpy(np.ascontiguousarray(v)).to(dev) for k, v in p["spacing"].items()}
    fx, sx = (sp[k + "x"].view(-1, 1, 1) for k in ("fd", "sd"))
    fy, sy = (sp[k + "y"].view(1, -1, 1) for k in ("fd", "sd"))
    fz, sz = (sp[k + "z"].view(1, 1, -1) for k in ("fd", "sd"))
    fx0, fy0, fz0, sx0, sy0, sz0 = (float(t.flatten()[0]) for t in (fx, fy, fz, sx, sy, sz))
    inner = ids[1:-1, 1:-1, :-1]
    C = [rows[q][inner] for q in range(9)]
    # shears: the sample one layer down, except in the z = 0 row
    down = torch.cat([ids[:, :, :1], ids[:, :, 2:]], 2)
    C4, C5, C6 = rows[9][down[1:-1, 1:]], rows[10][down[1:, 1:-1]], rows[11][ids[1:, 1:, :-1]]
    qx, qy = dt * dt / rows[12][ids[1:, 1:-1, :-1]], dt * dt / rows[12][ids[1:-1, 1:, :-1]]
    qz = dt * dt / rows[12][down[1:-1, 1:-1]]
    del inner, down
    vl = math.sqrt(p["table"][p["ids"][0, 0, 0], 0] / p["table"][p["ids"][0, 0, 0], 12]) * dt
    vt = math.sqrt(p["table"][p["ids"][0, 0, 0], 9] / p["table"][p["ids"][0, 0, 0], 12]) * dt

    def coef(v, d):
        return (v - d) / (v + d)

    walls = {"x": [coef(vl, float(sx.flatten()[-1]))] + [coef(vt, float(fx.flatten()[-1]))] * 2}
    for ax, f, s, own in (("y", fy, sy, 1), ("z", fz, sz, 2)):
        for end, at in (("0", 0), ("N", -1)):
            walls[ax + end] = [coef(vl, float(s.flatten()[at])) if c == own else coef(vt, float(f.flatten()[at]))
                               for c in range(3)]

    def zeros():
        return [torch.zeros(nx - (c == 0), ny - (c == 1), nz - (c == 2), dtype=torch.float64, device=dev)
                for c in range(3)]

    old, cur, new = zeros(), zeros(), zeros()
    T1, T2, T3 = (torch.zeros(nx, ny, nz, dtype=torch.float64, device=dev) for _ in range(3))
    T4 = torch.zeros(nx - 2, ny - 1, nz - 1, dtype=torch.float64, device=dev)
    T5 = torch.zeros(nx - 1, ny - 2, nz - 1, dtype=torch.float64, device=dev)
    T6 = torch.zeros(nx - 1, ny - 1, nz - 1, dtype=torch.float64, device=dev)
    surface = []
    for tt, s in enumerate(p["source"]):
        ux, uy, uz = cur
        if p["source_mode"] == "wall":
            uz[0] = float(s)
        else:
            uz[0, :, 0] = float(s)
        # strains and stresses (z = 0: first spacings, uz below the surface is 0)
        d1 = ux[1:, 1:-1, :-1] - ux[:-1, 1:-1, :-1]
        d2 = uy[1:-1, 1:, :-1] - uy[1:-1, :-1, :-1]
        d3 = torch.cat([uz[1:-1, 1:-1, :1], uz[1:-1, 1:-1, 1:] - uz[1:-1, 1:-1, :-1]], 2)
        e1, e2 = d1 / sx, d2 / sy
        e3 = torch.cat([d3[:, :, :1] / sz0, d3[:, :, 1:] / sz], 2)
        e1[:, :, 0], e2[:, :, 0] = d1[:, :, 0] / sx0, d2[:, :, 0] / sy0
        for q, T in enumerate((T1, T2, T3)):
            T[1:-1, 1:-1, :-1] = C[3 * q] * e1 + C[3 * q + 1] * e2 + C[3 * q + 2] * e3
        T3[:, :, 0] = 0

        def shear(T, c, a, ia, ia0, b, ib, ib0):
            T[:] = c * (a / ia + b / ib)
            T[:, :, 0] = c[:, :, 0] * (a[:, :, 0] / ia0 + b[:, :, 0] / ib0)

        shear(T4, C4, uy[1:-1, :, 1:] - uy[1:-1, :, :-1], fz, fy0, uz[1:-1, 1:] - uz[1:-1, :-1], fy, fz0)
        shear(T5, C5, ux[:, 1:-1, 1:] - ux[:, 1:-1, :-1], fz, fx0, uz[1:, 1:-1] - uz[:-1, 1:-1], fx, fz0)
        shear(T6, C6, (ux[:, 1:] - ux[:, :-1])[:, :, :-1], fy, fx0, (uy[1:] - uy[:-1])[:, :, :-1], fx, fz0)

        # divergences
        def div(a, ia, ia0, b, ib, ib0, z):
            d = a / ia + b / ib
            d[:, :, 0] = a[:, :, 0] / ia0 + b[:, :, 0] / ib0 + z[:, :, 0] / sz0
            d[:, :, 1:] += (z[:, :, 1:] - z[:, :, :-1]) / sz
            return d

        dx = div((T1[1:] - T1[:-1])[:, 1:-1, :-1], fx, fx0, T6[:, 1:] - T6[:, :-1], sy, sy0, T5)
        dy = div(T6[1:] - T6[:-1], sx, sx0, (T2[:, 1:] - T2[:, :-1])[1:-1, :, :-1], fy, fy0, T4)
        a, b = T5[1:] - T5[:-1], T4[:, 1:] - T4[:, :-1]
        t = (T3[1:-1, 1:-1, 1:] - T3[1:-1, 1:-1, :-1]) / fz
        dz = a / sx + b / sy + t
        last = t[:, :, 0] * fz0 if p["surface_mode"] == "reference" else t[:, :, 0]
        dz[:, :, 0] = a[:, :, 0] / sx0 + b[:, :, 0] / sy0 + last
        for c, (at, q, d) in enumerate((((slice(None), slice(1, -1), slice(-1)), qx, dx),
                                        ((slice(1, -1), slice(None), slice(-1)), qy, dy),
                                        ((slice(1, -1), slice(1, -1), slice(None)), qz, dz))):
            new[c][at] = 2 * cur[c][at] - old[c][at] + q * d
            u, n = cur[c], new[c]
            if p["bc"] == "rigid":
                n[-1], n[:, 0], n[:, -1], n[:, :, -1] = 0, 0, 0, 0
            else:
                n[-1] = u[-2] + walls["x"][c] * (n[-2] - u[-1])
                n[:, 0] = u[:, 1] + walls["y0"][c] * (n[:, 1] - u[:, 0])
                n[:, -1] = u[:, -2] + walls["yN"][c] * (n[:, -2] - u[:, -1])
                n[:, :, -1] = u[:, :, -2] + walls["zN"][c] * (n[:, :, -2] - u[:, :, -1])
        # points that a step does not write keep their value
        for c in range(3):
            old[c].copy_(cur[c])
            cur[c].copy_(new[c])
        if (tt + 1) % every == 0:
            surface.append(cur[2][:, :, 0].clone())
    return torch.stack(surface) if surface else torch.zeros(0, nx, ny, dtype=torch.float64, device=dev), cur


def _energy(case, seed):
    f, dt = _state_fields(case, seed)
    ids = torch.from_numpy(_crystal(case, seed)["ids"]).cuda().long()
    rows = torch.from_numpy(TABLE).cuda()
    u = [f[k].double() for k in FIELDS]
    v = [(u[c] - f[k + "_old"]) / dt if case["precision"] == "f64" else f["v" + k[1]].double()
         for c, k in enumerate(FIELDS)]

    def mat(q, at):
        return rows[:, q][at]

    kinetic = sum(float((mat(12, at) * w * w).sum()) for at, w in (
        (ids[1:-1, 1:-1, :-1], v[0][:-1, 1:-1, :-1]), (ids[1:-1, 2:-1, :-1], v[1][1:-1, 1:-1, :-1]),
        (ids[1:-1, 1:-1, 1:-1], v[2][1:-1, 1:-1, :-1])))
    e = [(u[0][1:] - u[0][:-1])[:, 1:-1, 1:-1] / DX, (u[1][:, 1:] - u[1][:, :-1])[1:-1, :, 1:-1] / DX,
         (u[2][:, :, 1:] - u[2][:, :, :-1])[1:-1, 1:-1] / DX]
    inner, strain = ids[1:-1, 1:-1, 1:-1], 0.0
    for a in range(3):
        for b in range(3):
            strain += float((mat(3 * a + b, inner) * e[a] * e[b]).sum())
    g = ((u[1][:, :, 1:] - u[1][:, :, :-1])[1:-1, :, 1:] + (u[2][:, 1:] - u[2][:, :-1])[1:-1, :, 1:]) / DX
    strain += float((mat(9, ids[1:-1, 1:, 2:]) * g * g).sum())
    g = ((u[0][:, :, 1:] - u[0][:, :, :-1])[:, 1:-1, 1:] + (u[2][1:] - u[2][:-1])[:, 1:-1, 1:]) / DX
    strain += float((mat(10, ids[1:, 1:-1, 2:]) * g * g).sum())
    g = ((u[0][:, 1:] - u[0][:, :-1])[:, :, 1:-1] + (u[1][1:] - u[1][:-1])[:, :, 1:-1]) / DX
    strain += float((mat(11, ids[1:, 1:, 1:-1]) * g * g).sum())
    return {"kinetic": 0.5 * kinetic, "strain": 0.5 * strain}


def exact(case, seed):
    kind = case["kind"]
    if kind == "energy":
        return _energy(case, seed)
    if kind == "batch":
        out = []
        for c, s in _instances(case, seed):
            surface, u = _leapfrog(_crystal(c, s), case["record_every"])
            out.append({"surface": surface, "uz": u[2]})
        return out
    if kind == "plugin":
        cyl, f = _inclusions(case, seed)
        nodes = (case["nx"] + 1, case["ny"] + 1, case["nz"] + 1)
        table = np.array([[np.array(m["c"])[a, b] * 1e10 for a, b in
                           [(0, 0), (0, 1), (0, 2), (1, 0), (1, 1), (1, 2), (2, 0), (2, 1), (2, 2), (3, 3), (4, 4),
                            (5, 5)]] + [m["p"]] for m in (GAAS, GOLD)])
        ids = np.zeros(nodes, np.uint8)
        x, y = np.arange(nodes[0])[:, None], np.arange(nodes[1])[None]
        for cx, cy, r in cyl:
            ids[(x - cx) ** 2 + (y - cy) ** 2 < r * r, : case["nz"] // 2 + 1] = 1
        sp = {k + a: np.ones(n - (k == "sd")) for k in ("fd", "sd") for a, n in
              zip("xyz", (case["nx"], case["ny"], case["nz"]))}
        fastest = max(math.sqrt(table[m, q] / table[m, 12]) for m in range(2) for q in (0, 9))
        dt = 0.5 / fastest
        p = {"spacing": sp, "ids": ids, "table": table, "dt": dt, "surface_mode": case["surface_mode"],
             "bc": "absorbing", "source_mode": "line",
             "source": np.sin(2 * np.pi * f * dt * np.arange(case["steps"]))}
    else:
        p = _crystal(case, seed)
    surface, u = _leapfrog(p, case["record_every"])
    return {"surface": surface, "ux": u[0], "uy": u[1], "uz": u[2]}
