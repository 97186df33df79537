"""Performance cases: the work a simulation program has this framework do, through its public calls.

Each case is one domain (or an ensemble of blocks) built and released the way a program builds it,
and one pass is what such a program does again and again: set a new run going and read its result
(halls, ensembles, scenes), or take the running simulation a stretch further and read the field
(blocks, cavities). Every pass ends with the field on the host and the books (the ledger), and every
timestep is audited as `Simulation::advance` audits it, but where open walls let energy out.

`listed` gives the cases, `draw` more of the same ranges, `prepare` the state, `run` one pass,
`work` its least bytes and operations, and `exact` the same outputs in 64 bits by plain torch.
"""
import math
import random

import numpy as np
import torch

from pantometry_b200 import domains, scenes

AIR = dict(speed=343.0, density=1.2)
C0 = 1.0 / math.sqrt(domains.EPSILON_0 * domains.MU_0)
SIGMA_SB = 5.670374419e-8  # W/m²K⁴
F64 = torch.float64


def listed():
    """Twelve cases: the smallest calls, ordinary runs and the largest, in both precisions."""
    return [
        # A small world scene, a hot spot in a 9³ block: 11 frames of one or a few substeps each, a
        # ledger a frame. Launches and the host's round trips are the whole of it.
        dict(name="scene_block", kind="scene", domain="block", size=9, frames=11, precision="f64"),
        # A clap in the corner of a 4.4 m room at 101 nodes across: 17 frames of about 20 substeps.
        dict(name="scene_room", kind="scene", domain="room", size=101, frames=17, precision="f64"),
        # The 64³ conduction block with Dirichlet faces, 1000 steps: resident in L2, bound by latency.
        dict(name="heat_f64_64", kind="block", nx=64, ny=64, nz=64, films="dirichlet", layout="uniform",
             precision="f64", steps=1000),
        # A uniform block larger than L2 with convective films, bit-exact form.
        dict(name="heat_f64_256", kind="block", nx=256, ny=240, nz=224, films="convective", layout="uniform",
             precision="f64", steps=400),
        # The same physics with FP32 fields at the size of the block benchmark.
        dict(name="heat_f32_256", kind="block", nx=256, ny=256, nz=256, films="dirichlet", layout="uniform",
             precision="f32", steps=1200),
        # A part of two materials with a dissipating chip, cooled by air on every face, its surfaces
        # radiating: ragged extents, per-cell coefficients, a step limit that follows the state.
        dict(name="heat_f64_part", kind="block", nx=150, ny=121, nz=93, films="radiating", layout="filled",
             precision="f64", steps=300),
        # The acoustic hall of the benchmark: 256³ nodes, noise, a Ricker source, FP32 fields.
        dict(name="hall_f32_256", kind="hall", nx=256, ny=256, nz=256, precision="f32", source=True, block=0,
             steps=1000),
        # An ordinary hall of odd extents in the bit-exact form.
        dict(name="hall_f64_ragged", kind="hall", nx=143, ny=101, nz=79, precision="f64", source=True, block=0,
             steps=500),
        # The vacuum cavity of the benchmark, conducting walls and a dipole: the largest case.
        dict(name="cavity_f32_384", kind="cavity", nx=384, ny=384, nz=384, medium="vacuum", walls="conducting",
             precision="f32", steps=200),
        # A cavity with dielectric inclusions in a tenth of its cells.
        dict(name="cavity_f32_dielectric", kind="cavity", nx=128, ny=128, nz=128, medium="dielectric",
             walls="conducting", precision="f32", steps=800),
        # An open box of odd extents around a metal obstacle, bit-exact form.
        dict(name="cavity_f64_open", kind="cavity", nx=101, ny=83, nz=67, medium="obstacle", walls="open",
             precision="f64", steps=300),
        # An ensemble of uneven blocks, 16 to 128 cells an axis, FP32 fields.
        dict(name="ensemble_f32", kind="ensemble", blocks=160, lo=16, hi=128, precision="f32", steps=400),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _extents(rng, lo, hi):
    """Three extents about one size, odd ones and multiples of 32 among them."""
    n = _log(rng, lo, hi)
    out = [min(hi, max(lo, int(n * rng.uniform(0.7, 1.3)))) for _ in range(3)]
    how = rng.random()
    if how < 0.35:
        out = [max(lo, (v // 32) * 32) if v >= 32 else v for v in out]
    elif how < 0.6:
        out[0] = max(lo, (out[0] // 4) * 4)
    return out


def _steps(rng, cells, ns_per_cell):
    """Enough steps for a pass of some 20 to 60 ms at `ns_per_cell`, within 64 to 1500."""
    return max(64, min(1500, int(rng.uniform(2e7, 6e7) / (cells * ns_per_cell + 3000.0))))


def draw(rng):
    """One more case: the listed ones' kinds, sizes, precisions, films, media and walls, mixed anew."""
    kind = rng.choice(["scene", "block", "block", "block", "hall", "hall", "cavity", "cavity", "ensemble"])
    precision = rng.choice(["f64", "f32"])
    if kind == "scene":
        what = rng.choice(["block", "room"])
        size = rng.randint(6, 24) if what == "block" else _log(rng, 41, 241)
        return dict(kind=kind, domain=what, size=size, frames=rng.randint(9, 24), precision=precision)
    if kind == "block":
        nx, ny, nz = _extents(rng, 24, 256)
        layout = rng.choice(["uniform", "uniform", "filled"])
        films = rng.choice(["none", "dirichlet", "convective", "radiating"])
        if layout == "filled":
            nx, ny, nz = min(nx, 160), min(ny, 160), min(nz, 160)
            films = "convective" if films == "dirichlet" or (films == "radiating" and precision == "f32") else films
        cost = 0.012 if precision == "f64" else 0.005  # ns a cell and step, about
        cost *= (4.0 if layout == "filled" else 1.0) * (2.0 if films in ("convective", "radiating") else 1.0)
        steps = _steps(rng, nx * ny * nz, cost)
        return dict(kind=kind, nx=nx, ny=ny, nz=nz, films=films, layout=layout, precision=precision, steps=steps)
    if kind == "hall":
        nx, ny, nz = _extents(rng, 24, 256)
        steps = _steps(rng, nx * ny * nz, 0.012 if precision == "f64" else 0.006)
        return dict(kind=kind, nx=nx, ny=ny, nz=nz, precision=precision, source=rng.random() < 0.6,
                    block=rng.choice([0, 0, 0, 8, 32]), steps=steps)
    if kind == "cavity":
        nx, ny, nz = _extents(rng, 24, 256)
        medium = rng.choice(["vacuum", "dielectric", "obstacle", "lossy"])
        walls = rng.choice(["conducting", "conducting", "open"])
        cost = 0.025 if precision == "f64" else 0.012
        steps = _steps(rng, nx * ny * nz, cost * (1.5 if walls == "open" or medium != "vacuum" else 1.0))
        return dict(kind=kind, nx=nx, ny=ny, nz=nz, medium=medium, walls=walls, precision=precision, steps=steps)
    hi = _log(rng, 32, 128)
    blocks = max(4, min(256, int(4e7 / (0.4 * (hi + 16)) ** 3 * rng.uniform(0.2, 1.0))))
    return dict(kind=kind, blocks=blocks, lo=16, hi=hi, precision=precision, steps=rng.randint(100, 200))


# ---- inputs --------------------------------------------------------------------------------------

def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed) & 0x7FFFFFFF)


def _pinned(t):
    """A pinned host array holding the values of a device tensor, or room for them."""
    host = torch.empty(t.numel(), dtype=F64, pin_memory=True)
    host.copy_(t.reshape(-1))
    return host.numpy()


def _room_for(n):
    return torch.empty(n, dtype=F64, pin_memory=True).numpy()


def _hot_spot(counts, centre, amplitude, sigma, base):
    nx, ny, nz = counts
    i, j, k = (torch.arange(n, dtype=F64, device="cuda") + 0.5 - c for n, c in zip(counts, centre))
    r2 = k[:, None, None] ** 2 + j[None, :, None] ** 2 + i[None, None, :] ** 2
    return base + amplitude * torch.exp(-r2 / (2.0 * sigma * sigma))


ALPHA_BLOCK = dict(density=1000.0, conductivity=100.0, specific_heat=1000.0, emissivity=0.0)


def _block_inputs(case, seed):
    """A block's materials, fill mask, chip mask and watts, films and initial kelvin."""
    r = random.Random(seed)
    counts = nx, ny, nz = case["nx"], case["ny"], case["nz"]
    dx = 1e-3
    emits = case["films"] == "radiating"
    aluminium = dict(scenes.ALUMINIUM_6061, emissivity=0.09 if emits else 0.0)
    glass = dict(scenes.BOROSILICATE_CROWN, emissivity=0.90 if emits else 0.0)
    filled = case["layout"] == "filled"
    bulk = aluminium if filled or emits else ALPHA_BLOCK
    fill = chip = None
    if filled:
        k = np.arange(nz)[:, None, None]
        j = np.arange(ny)[None, :, None]
        i = np.arange(nx)[None, None, :]
        cut = int(nz * r.uniform(0.4, 0.6))
        fill = np.broadcast_to(k >= cut, (nz, ny, nx)).astype(np.uint8).reshape(-1)
        lo = [int(v * r.uniform(0.2, 0.4)) for v in counts]
        inside = [(q >= a) & (q < a + max(1, v // 4)) for q, a, v in zip((i, j, k), lo, counts)]
        chip = np.broadcast_to(inside[0] & inside[1] & inside[2], (nz, ny, nx)).astype(np.uint8).reshape(-1)
    films = []
    for f in range(6):
        area = [ny * nz, ny * nz, nx * nz, nx * nz, nx * ny, nx * ny][f] * dx * dx
        if case["films"] == "dirichlet":
            films.append((f, 300.0, math.inf, area))
        elif case["films"] in ("convective", "radiating"):
            films.append((f, 300.0 + r.uniform(-8.0, 8.0), r.uniform(10.0, 60.0), area))
    centre = [n / 2 + r.uniform(-0.1, 0.1) * n for n in counts]
    cells = _hot_spot(counts, centre, 50.0, max(2.0, min(counts) / 8.0), 300.0)
    return dict(counts=counts, dx=dx, bulk=bulk, glass=glass, fill=fill, chip=chip, watts=r.uniform(2.0, 8.0),
                films=films, cells=cells, initial=300.0)


def _block_dt(case, limit):
    """Under the opening limit with room for a radiating surface that warms."""
    return 0.9 * limit


def _hall_inputs(case, seed):
    r = random.Random(seed)
    g = _gen(seed)
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    dx = 5e-3
    p = (torch.rand((nz, ny, nx), dtype=F64, device="cuda", generator=g) * 2.0 - 1.0) * 1e-3
    speeds = None
    fastest = AIR["speed"]
    if case["block"]:
        nb = [-(-n // case["block"]) for n in (nx, ny, nz)]
        speeds = np.array([r.uniform(300.0, 1500.0) for _ in range(nb[0] * nb[1] * nb[2])])
        fastest = float(speeds.max())
    dx_eff = max((nx - 1) * dx / (nx - 1), np.finfo(np.float64).tiny)
    dt = 0.5 * dx_eff / (fastest * math.sqrt(3.0))
    source = None
    if case["source"]:
        t = (np.arange(case["steps"], dtype=np.float64) + 1.0) * dt
        f = r.uniform(1500.0, 2500.0)
        a = (math.pi * f * (t - 1.2 / f)) ** 2
        at = [int(n * r.uniform(0.3, 0.7)) for n in (nx, ny, nz)]
        source = (at, r.uniform(0.5, 1.5) * (1.0 - 2.0 * a) * np.exp(-a))
    return dict(p=p, speeds=speeds, dt=dt, source=source, dx=dx, fastest=fastest)


def _cavity_inputs(case, seed):
    r = random.Random(seed)
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    dx = 1e-3
    dt = 0.99 * (0.5773502691896258 * dx / C0)
    f0 = C0 / (r.uniform(18.0, 24.0) * dx)
    tau = 1.0 / (math.pi * 0.5 * f0)
    t0 = 4.0 * tau
    t = (np.arange(case["steps"], dtype=np.float64) + 0.5) * dt
    current = r.uniform(0.5, 1.5) / (dx * dx) * np.exp(-(((t - t0) / tau) ** 2)) * np.sin(2.0 * math.pi * f0 * t)
    at = [int(n * r.uniform(0.4, 0.6)) for n in (nx, ny, nz)]
    eps = solid = None
    sigma = 0.0
    if case["medium"] == "dielectric":
        g = _gen(seed)
        pick = torch.rand((nz, ny, nx), dtype=F64, device="cuda", generator=g) < 0.1
        eps = torch.where(pick, 1.0 + 3.0 * torch.rand((nz, ny, nx), dtype=F64, device="cuda", generator=g), 1.0)
    elif case["medium"] == "obstacle":
        solid = np.zeros((nz, ny, nx), dtype=np.uint8)
        lo = [int(n * 0.15) for n in (nx, ny, nz)]
        hi = [max(a + 1, int(n * r.uniform(0.25, 0.33))) for a, n in zip(lo, (nx, ny, nz))]
        solid[lo[2]:hi[2], lo[1]:hi[1], lo[0]:hi[0]] = 1
    elif case["medium"] == "lossy":
        sigma = r.uniform(0.005, 0.05)
    # a closed vacuum cavity also rings in one of its own modes
    mode = (r.randint(1, 3), r.randint(1, 3)) if case["medium"] == "vacuum" and case["walls"] == "conducting" else None
    return dict(dx=dx, dt=dt, current=current, at=at, eps=eps, solid=solid, sigma=sigma, mode=mode)


def _ensemble_inputs(case, seed):
    r = random.Random(seed)
    shape = random.Random(case["blocks"] * 1009 + case["hi"])  # the blocks' extents: the case's own
    grids, cells = [], []
    for _ in range(case["blocks"]):
        counts = tuple(shape.randint(case["lo"], case["hi"]) for _ in range(3))
        alpha = 10.0 ** r.uniform(-6.0, -3.0)
        centre = [r.uniform(0.0, n) for n in counts]
        cells.append(_hot_spot(counts, centre, 50.0, min(8.0, min(counts) / 8.0), 300.0))
        grids.append({"counts": counts, "dx": 1e-3, "initial": 300.0, "convection": math.inf,
                      "substance": dict(density=1000.0, conductivity=alpha * 1e6, specific_heat=1000.0,
                                        emissivity=0.0)})
    return grids, cells


def _scene(case, seed):
    """A world scene of one domain, as the reference's scene files write them."""
    r = random.Random(seed)
    n = case["size"]
    if case["domain"] == "block":
        d = {"kind": "block", "name": "block", "cells": [n, n, n], "cell_mm": 1.0, "initial_c": 20.0,
             "hot_spot": {"at": [r.randrange(n) for _ in range(3)], "above_k": r.uniform(40.0, 80.0)}}
        duration, tol = 0.006 * case["frames"] / 11.0, 1e-9 if case["precision"] == "f64" else 1e-6
    else:
        d = {"kind": "room", "name": "room", "width_m": 4.4, "height_m": 3.1, "cells_across": n,
             "release": {"as": "pulse", "amplitude_pa": r.uniform(0.5, 1.5), "radius_m": 0.22,
                         "x_m": r.uniform(0.7, 1.4), "y_m": r.uniform(0.6, 1.2)}}
        duration, tol = 0.03 * case["frames"] / 17.0, 1e-6
    return {"schedule": "multirate", "duration_s": duration, "frames": case["frames"],
            "conservation_tolerance": tol, "domains": [d]}


def prepare(case, seed):
    kind, precision = case["kind"], case["precision"]
    if kind == "scene":
        scene = _scene(case, seed)
        dom = scenes.build(scene, precision=precision)
        d = scene["domains"][0]
        if case["domain"] == "block":
            start = scenes.block_layout(d)[2]
        else:
            start = scenes.room_release(dom.cells, dom.dx, d["release"])
        return dict(case=case, scene=scene, dom=dom, start=start)
    if kind == "block":
        q = _block_inputs(case, seed)
        m = q["bulk"]
        b = domains.Solid3D(q["counts"], q["dx"], m["density"], m["conductivity"], m["specific_heat"], q["initial"],
                            emissivity=m["emissivity"], precision=precision)
        if q["fill"] is not None:
            s = q["glass"]
            b.fill(q["fill"], s["density"], s["conductivity"], s["specific_heat"], s["emissivity"])
            b.dissipating(q["watts"], q["chip"])
        for face, ambient, h, area in q["films"]:
            b.losing_from(face, ambient, h, area)
        b.cells = _pinned(q["cells"])
        b.set_tolerance(1e-9 if precision == "f64" else 1e-6)
        return dict(case=case, dom=b, dt=_block_dt(case, b.max_stable_dt()))
    if kind == "hall":
        q = _hall_inputs(case, seed)
        nx, ny, nz = case["nx"], case["ny"], case["nz"]
        h = domains.Hall((nx - 1) * q["dx"], (ny - 1) * q["dx"], (nz - 1) * q["dx"], nx, AIR["speed"],
                         AIR["density"], precision=precision)
        assert h.nodes == (nx, ny, nz)
        if q["speeds"] is not None:
            h.set_speed_blocks(case["block"], q["speeds"])
        if q["source"] is not None:
            (i, j, k), wave = q["source"]
            h.set_source(i + nx * (j + ny * k), wave)
        h.set_tolerance(1e-9 if precision == "f64" else 1e-6)
        return dict(case=case, dom=h, dt=q["dt"], p=_pinned(q["p"]), out=_room_for(h.n))
    if kind == "cavity":
        q = _cavity_inputs(case, seed)
        nx, ny, nz = case["nx"], case["ny"], case["nz"]
        c = domains.Cavity((nx, ny, nz), q["dx"], sigma=q["sigma"], precision=precision)
        if q["eps"] is not None:
            c.fill_cells(eps_r=_pinned(q["eps"]))
        if q["solid"] is not None:
            c.obstruct(q["solid"])
        if case["walls"] == "open":
            for w in domains.WALLS:
                c.set_boundary(w, "open")
        if q["mode"] is not None:
            c.release_mode(q["mode"], 100.0, q["dt"])
        i, j, k = q["at"]
        c.set_source(i + (nx + 1) * (j + (ny + 1) * k), q["current"])
        # energy leaves through open walls and into a lossy medium's swinging books: no audit there
        audited = case["walls"] == "conducting" and case["medium"] != "lossy"
        c.set_tolerance((1e-9 if precision == "f64" else 1e-5) if audited else -1.0)
        return dict(case=case, dom=c, dt=q["dt"], out=_room_for(c.shapes()["ez"]))
    grids, cells = _ensemble_inputs(case, seed)
    for g, limit in zip(grids, domains.Ensemble.max_stable_dt(grids)):
        g["dt"] = 0.9 * float(limit)
    e = domains.Ensemble(grids, precision=precision)
    start = _pinned(torch.cat([c.reshape(-1) for c in cells]))
    e.upload(start)
    e.set_tolerance(1e-9 if precision == "f64" else 1e-6)
    e.autotune()
    return dict(case=case, dom=e, start=start, out=_room_for(e.n))


def _held(violation):
    if violation is not None:
        raise RuntimeError(f"the step was refused or its audit failed: {violation}")


def run(state):
    case, dom = state["case"], state["dom"]
    kind, steps = case["kind"], case.get("steps")
    if kind == "scene":  # one run of the scene, from its release to its last frame
        if case["domain"] == "block":
            dom.cells = state["start"]
        else:
            dom.release(state["start"])
        got = scenes.run(state["scene"], dom)
        _held(got["violation"])
        field = dom.cells if case["domain"] == "block" else dom.fields()["p"]
        return {"field": field, "totals": np.array([f["total"] for f in got["frames"]])}
    if kind == "block":  # `steps` more, then the field and the books
        _held(dom.step(state["dt"], steps))
        return {"field": dom.cells, "books": np.array(dom.ledger()["parts"])}
    if kind == "hall":  # a run from a fresh release
        dom.release(state["p"])
        _held(dom.step(state["dt"], steps))
        return {"field": dom.download_pressure(state["out"]), "books": np.array(dom.ledger()["parts"][:3])}
    if kind == "cavity":  # `steps` more, then the component along the dipole and the books
        _held(dom.step(state["dt"], steps))
        return {"field": dom.download_component("ez", state["out"]), "books": np.array(dom.ledger()["parts"])}
    dom.upload(state["start"])  # a run of every block from a fresh state
    _held(dom.step(steps))
    books = np.array([led["parts"] for led in dom.ledgers()])
    return {"field": dom.download(state["out"]), "books": books}


# ---- least work ----------------------------------------------------------------------------------

def _substeps(scene, limit):
    return scenes.substeps_for(scenes.window(scene), limit)


def work(case):
    """Each timestep reads and writes every field once (and reads the coefficients that vary), each
    pass moves its inputs and results across the host's link; operations counted per cell-update."""
    kind = case["kind"]
    e = 8 if case["precision"] == "f64" else 4
    if kind == "scene":
        n = case["size"]
        scene = _scene(case, 1)
        if case["domain"] == "block":
            m = scenes.ALUMINIUM_6061
            limit = 1e-6 * m["density"] * m["specific_heat"] / m["conductivity"] / 6.0
            cells, per, ops = n ** 3, 2 * e, 24
        else:
            dx = 4.4 / (n - 1)
            limit = dx / (scenes.AIR["speed"] * math.sqrt(2.0))
            cells, per, ops = n * (round(3.1 / dx) + 1), 6 * e, 18
        steps = case["frames"] * _substeps(scene, limit)
        return {"bytes": steps * cells * per + 16 * cells, "flops": steps * cells * ops}
    steps = case["steps"]
    if kind == "block":
        cells = case["nx"] * case["ny"] * case["nz"]
        per = 2 * e + (0 if case["layout"] == "uniform" else 4 * e + 8)  # three faces, mobility, capacity
        return {"bytes": cells * (steps * per + 8), "flops": steps * cells * 24}
    if kind == "hall":
        cells = case["nx"] * case["ny"] * case["nz"]
        return {"bytes": cells * (steps * 8 * e + 16), "flops": steps * cells * 30}
    if kind == "cavity":
        cells = case["nx"] * case["ny"] * case["nz"]
        per = 12 * e + (3 * e if case["medium"] == "dielectric" else 0)
        return {"bytes": cells * (steps * per + 8), "flops": steps * cells * 54}
    shape = random.Random(case["blocks"] * 1009 + case["hi"])
    cells = 0
    for _ in range(case["blocks"]):
        a, b, c = (shape.randint(case["lo"], case["hi"]) for _ in range(3))
        cells += a * b * c
    return {"bytes": cells * (steps * 2 * e + 16), "flops": steps * cells * 24}


# ---- the same outputs in 64 bits -----------------------------------------------------------------

def _series(film, half):
    return 1.0 / (1.0 / film + 1.0 / half) if film > 0.0 else 0.0


def _exact_heat(t, dx, k, cap, films, dt, steps, initial, src=None, eps=None, per_step=None):
    """Explicit conduction with films on the faces: t, k and cap of shape (nz, ny, nx) (k and cap may
    be numbers); films as (face, ambient, h, share); src in watts, eps the emissivity. Returns the
    field and (stored, lost, -supplied)."""
    t = t.clone()
    cap_t = torch.as_tensor(cap, dtype=F64, device=t.device)
    uniform = not torch.is_tensor(k)
    faces = {}
    if not uniform:
        for ax in range(3):
            n = k.shape[ax]
            a, b = k.narrow(ax, 0, n - 1), k.narrow(ax, 1, n - 1)
            faces[ax] = 2.0 * a * b / (a + b)
    mob = dx / cap_t
    supplied = 0.0
    lost_t = torch.zeros((), dtype=F64, device=t.device)
    totals = []
    done = 0
    for count in (per_step or [steps]):
        for _ in range(count):
            flux = torch.zeros_like(t)
            for ax in (2, 1, 0):
                n = t.shape[ax]
                if n < 2:
                    continue
                d = t.narrow(ax, 1, n - 1) - t.narrow(ax, 0, n - 1)
                d = d * (k if uniform else faces[ax])
                flux.narrow(ax, 0, n - 1).add_(d)
                flux.narrow(ax, 1, n - 1).sub_(d)
            shed = None
            if films:
                shed = torch.zeros_like(t)
                for f, ambient, h, share in films:
                    ax = 2 - f // 2
                    at = 0 if f % 2 == 0 else t.shape[ax] - 1
                    here = t.select(ax, at)
                    kc = k if uniform else k.select(ax, at)
                    half = 2.0 * kc * share / dx
                    gap = here - ambient
                    if math.isinf(h):
                        g = half
                    else:
                        bare = h * share
                        if eps is not None:
                            ec = eps if not torch.is_tensor(eps) else eps.select(ax, at)
                            bare = bare + ec * SIGMA_SB * share * (here ** 2 + ambient ** 2) * (here + ambient)
                        g = 1.0 / (1.0 / bare + 1.0 / half)
                    shed.select(ax, at).add_(g * gap / dx)
                lost_t += (dt * mob * cap_t * shed).sum()
                flux -= shed
            t += dt * mob * flux
            if src is not None:
                t += src * dt / cap_t
            done += 1
        totals.append(((t - initial) * cap_t).sum() + lost_t)
    if src is not None:
        supplied = float(src.sum()) * dt * done
    stored = float(((t - initial) * cap_t).sum())
    return t, (stored, float(lost_t), -supplied), [float(v) for v in totals]


def _exact_block(case, seed):
    q = _block_inputs(case, seed)
    dx, counts = q["dx"], q["counts"]
    nx, ny, nz = counts
    vol = dx * dx * dx
    m, s = q["bulk"], q["glass"]
    k, cap, eps, src = m["conductivity"], m["density"] * vol * m["specific_heat"], None, None
    if case["films"] == "radiating":
        eps = m["emissivity"]
    if q["fill"] is not None:
        mask = torch.from_numpy(q["fill"].reshape(nz, ny, nx)).cuda().bool()
        two = lambda a, b: torch.where(mask, torch.tensor(a, dtype=F64).cuda(), torch.tensor(b, dtype=F64).cuda())
        cap = two(s["density"] * vol * s["specific_heat"], cap)
        k = two(s["conductivity"], k)
        if eps is not None:
            eps = two(s["emissivity"], eps)
        chip = torch.from_numpy(q["chip"].reshape(nz, ny, nx)).cuda().to(F64)
        src = chip * (q["watts"] / float(chip.sum()))
    cells_on = [ny * nz, ny * nz, nx * nz, nx * nz, nx * ny, nx * ny]
    films = [(f, a, h, area / cells_on[f]) for f, a, h, area in q["films"]]
    t = q["cells"]
    # the limit max_stable_dt gives: 1 / max of mobility · (face conductivities + film loss / dx)
    full = torch.zeros_like(t)
    for ax in range(3):
        n = t.shape[ax]
        if n < 2:
            continue
        if torch.is_tensor(k):
            a, b = k.narrow(ax, 0, n - 1), k.narrow(ax, 1, n - 1)
            f = 2.0 * a * b / (a + b)
        else:
            f = k
        full.narrow(ax, 0, n - 1).add_(f)
        full.narrow(ax, 1, n - 1).add_(f)
    for f, ambient, h, share in films:
        ax = 2 - f // 2
        at = 0 if f % 2 == 0 else t.shape[ax] - 1
        half = 2.0 * (k.select(ax, at) if torch.is_tensor(k) else k) * share / dx
        if math.isinf(h):
            g = half
        else:
            hh = h
            if eps is not None:
                hot = torch.clamp(t.select(ax, at), min=ambient)
                hh = h + 4.0 * (eps.select(ax, at) if torch.is_tensor(eps) else eps) * SIGMA_SB * hot ** 3
            g = 1.0 / (1.0 / (hh * share) + 1.0 / half)
        full.select(ax, at).add_(g / dx)
    dt = _block_dt(case, 1.0 / float((full * (dx / cap)).max()))
    field, books, _ = _exact_heat(t, dx, k, cap, films, dt, case["steps"], q["initial"], src, eps)
    return {"field": field.reshape(-1), "books": np.array(books)}


def _face_weights(n, device):
    w = torch.ones(n, dtype=F64, device=device)
    w[0] = w[-1] = 2.0
    return w


def _exact_wave(p, dx, volume, rho, c, dt, steps, source=None, per_step=None):
    """The staggered acoustic scheme over p of shape (nz, ny, nx) or (ny, nx), rigid walls; c a speed or
    one per node. Returns the pressure, (invariant, offset, -injected) and the totals at `per_step`."""
    p = p.clone()
    dev, nd = p.device, p.dim()
    rc2 = rho * torch.as_tensor(c, dtype=F64, device=dev) ** 2
    wall = [_face_weights(n, dev).reshape([-1 if a == q else 1 for a in range(nd)]) for q, n in enumerate(p.shape)]
    share = 1.0
    for w in wall:
        share = share / w
    v = [torch.zeros([n - (1 if a == q else 0) for a, n in enumerate(p.shape)], dtype=F64, device=dev) for q in range(nd)]
    face_share = []
    for q in range(nd):
        s = torch.ones([1] * nd, dtype=F64, device=dev)
        for a in range(nd):
            if a != q:
                s = s / wall[a]
        face_share.append(s)

    def invariant(p, pp):
        total = (share * p * pp / (2.0 * rc2) * volume).sum()
        for q in range(nd):
            total = total + (face_share[q] * v[q] * v[q]).sum() * (0.5 * rho * volume)
        return float(total)

    datum = invariant(p, p)
    offset = injected = last = 0.0
    totals = []
    n = 0
    at = wn = None
    if source is not None:
        at = tuple(reversed(source[0]))
        rs = rc2[at] if rc2.dim() else rc2
        wn = float(share[at] * volume / (2.0 * rs))
    inj = torch.zeros((), dtype=F64, device=dev)
    for count in (per_step or [steps]):
        for _ in range(count):
            gain = (dt if n else 0.5 * dt) / (rho * dx)
            for q in range(nd):
                m = p.shape[q]
                v[q] -= gain * (p.narrow(q, 1, m - 1) - p.narrow(q, 0, m - 1))
            pp = p.clone()
            div = torch.zeros_like(p)
            for q in range(nd):
                m = p.shape[q]
                d = torch.zeros_like(p)
                d.narrow(q, 0, m - 1).add_(v[q])
                d.narrow(q, 1, m - 1).sub_(v[q])
                div += wall[q] * d
            p = p - dt * rc2 / dx * div
            immediate = 0.0
            if source is not None:
                delta = float(source[1][n]) if n < len(source[1]) else 0.0
                inj += wn * (last + delta) * pp[at]
                if n == 0:
                    immediate = wn * delta * float(pp[at])
                p[at] += delta
                last = delta
            if n == 0:
                offset = datum - (invariant(p, pp) - immediate)
            n += 1
        if per_step:
            totals.append(invariant(p, pp) + offset)
    injected = float(inj)
    return p, (invariant(p, pp), offset, -injected), [datum] + totals


def _exact_hall(case, seed):
    q = _hall_inputs(case, seed)
    c = AIR["speed"]
    if q["speeds"] is not None:
        b = case["block"]
        nb = [-(-n // b) for n in (case["nx"], case["ny"], case["nz"])]
        s = torch.from_numpy(q["speeds"].reshape(nb[2], nb[1], nb[0])).cuda()
        c = s
        for ax, n in enumerate((case["nz"], case["ny"], case["nx"])):
            c = c.repeat_interleave(b, ax).narrow(ax, 0, n)
    p, books, _ = _exact_wave(q["p"], q["dx"], q["dx"] ** 3, AIR["density"], c, q["dt"], case["steps"], q["source"])
    return {"field": p.reshape(-1), "books": np.array(books)}


def _edge_mean(cells, axes):
    """Mean of the four cells around each edge normal to `axes`, the outermost cells repeated."""
    for ax in axes:
        n = cells.shape[ax]
        pad = torch.cat([cells.narrow(ax, 0, 1), cells, cells.narrow(ax, n - 1, 1)], ax)
        cells = 0.5 * (pad.narrow(ax, 0, n + 1) + pad.narrow(ax, 1, n + 1))
    return cells


def _exact_cavity(case, seed):
    q = _cavity_inputs(case, seed)
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    dx, dt = q["dx"], q["dt"]
    dev = "cuda"
    E = [torch.zeros(s, dtype=F64, device=dev) for s in ((nz + 1, ny + 1, nx), (nz + 1, ny, nx + 1), (nz, ny + 1, nx + 1))]
    H = [torch.zeros(s, dtype=F64, device=dev) for s in ((nz, ny, nx + 1), (nz, ny + 1, nx), (nz + 1, ny, nx))]
    normal = [(0, 1), (0, 2), (1, 2)]  # the array axes (z, y, x) normal to each E edge
    if q["eps"] is not None:
        eps = [domains.EPSILON_0 * _edge_mean(q["eps"], ax) for ax in normal]
    else:
        eps = [domains.EPSILON_0] * 3
    mu, s = domains.MU_0, q["sigma"]

    def diff(f, ax):
        n = f.shape[ax]
        return f.narrow(ax, 1, n - 1) - f.narrow(ax, 0, n - 1)

    def magnetic(h):
        g = h / dx / mu
        H[0].sub_(g * (diff(E[2], 1) - diff(E[1], 0)))
        H[1].sub_(g * (diff(E[0], 0) - diff(E[2], 2)))
        H[2].sub_(g * (diff(E[1], 2) - diff(E[0], 1)))

    def inner(f, axes):
        for ax in axes:
            f = f.narrow(ax, 1, f.shape[ax] - 2)
        return f

    def weigh(f, axes):
        """f weighted by one half on each outermost plane of `axes`."""
        for ax in axes:
            w = torch.ones(f.shape[ax], dtype=F64, device=dev)
            w[0] = w[-1] = 0.5
            f = f * w.reshape([-1 if a == ax else 1 for a in range(3)])
        return f

    volume = dx * (dx * dx)
    started = False
    if q["mode"] is not None:
        m, pm = q["mode"]
        x = torch.arange(nx + 1, dtype=F64, device=dev) * dx
        z = torch.arange(nz + 1, dtype=F64, device=dev) * dx
        E[1] += 100.0 * torch.sin(math.pi * m / (nx * dx) * x)[None, None, :] * torch.sin(math.pi * pm / (nz * dx) * z)[:, None, None]
        E[1][:, :, 0] = E[1][:, :, -1] = 0.0
        E[1][0] = E[1][-1] = 0.0
        magnetic(-0.5 * dt)
        started = True
    solid = None
    if q["solid"] is not None:
        cells = torch.from_numpy(q["solid"]).to(dev).to(F64)
        solid = []
        for axes in normal:
            f = cells
            for ax in axes:
                n = f.shape[ax]
                zero = torch.zeros_like(f.narrow(ax, 0, 1))
                pad = torch.cat([zero, f, zero], ax)
                f = torch.maximum(pad.narrow(ax, 0, n + 1), pad.narrow(ax, 1, n + 1))
            solid.append(f > 0)
    kk = (C0 * dt - dx) / (C0 * dt + dx)
    i, j, k = q["at"]
    if not started:
        magnetic(0.5 * dt)
    dissipated = torch.zeros((), dtype=F64, device=dev)
    work_ = torch.zeros((), dtype=F64, device=dev)
    booked = 0.0
    inv = 0.0
    prev = None
    for n in range(case["steps"]):
        was = [h.clone() for h in H] if n + 1 == case["steps"] else None
        magnetic(dt)
        if was is not None:
            inv = sum(float(weigh(eps[c] * E[c] * E[c], normal[c]).sum()) for c in range(3)) * 0.5 * volume
            inv += sum(float(weigh(mu * H[c] * was[c], (2 - c,)).sum()) for c in range(3)) * 0.5 * volume
            booked = float(work_)
        curls = (lambda: diff(H[2], 1).narrow(0, 1, nz - 1) - diff(H[1], 0).narrow(1, 1, ny - 1),
                 lambda: diff(H[0], 0).narrow(2, 1, nx - 1) - diff(H[2], 2).narrow(0, 1, nz - 1),
                 lambda: diff(H[1], 2).narrow(1, 1, ny - 1) - diff(H[0], 1).narrow(2, 1, nx - 1))
        for c in range(3):
            e = inner(eps[c], normal[c]) if torch.is_tensor(eps[c]) else eps[c]
            half = s * dt / (2.0 * e)
            f = inner(E[c], normal[c])
            before = f.clone() if s else None
            at_src = float(E[2][k, j, i]) if c == 2 else 0.0
            f.mul_((1.0 - half) / (1.0 + half)).add_(curls[c]() * ((dt / (e * dx)) / (1.0 + half)))
            if c == 2:
                es = float(eps[2][k, j, i]) if torch.is_tensor(eps[2]) else eps[2]
                jn = float(q["current"][n]) if n < len(q["current"]) else 0.0
                E[2][k, j, i] -= (dt / es) / (1.0 + s * dt / (2.0 * es)) * jn
                work_ -= dt * volume * jn * 0.5 * (at_src + E[2][k, j, i])
            if s:
                dissipated += (s * (0.5 * (before + f)) ** 2).sum() * (dt * volume)
        if case["walls"] == "open":
            for w in range(6):
                ax = 2 - w // 2
                for c in range(3):
                    if ax not in normal[c]:
                        continue
                    last = E[c].shape[ax] - 1
                    edge, near = (0, 1) if w % 2 == 0 else (last, last - 1)
                    if prev is None:
                        E[c].select(ax, edge).zero_()
                    else:
                        E[c].select(ax, edge).copy_(prev[c].select(ax, near) + kk * (E[c].select(ax, near) - prev[c].select(ax, edge)))
            prev = [f.clone() for f in E]
        if solid is not None:
            for c in range(3):
                E[c].masked_fill_(solid[c], 0.0)
    return {"field": E[2].reshape(-1), "books": np.array([inv, float(dissipated), -booked])}


def exact(case, seed):
    kind = case["kind"]
    if kind == "block":
        return _exact_block(case, seed)
    if kind == "hall":
        return _exact_hall(case, seed)
    if kind == "cavity":
        return _exact_cavity(case, seed)
    if kind == "ensemble":
        grids, cells = _ensemble_inputs(case, seed)
        fields, books = [], []
        for g, t in zip(grids, cells):
            k = g["substance"]["conductivity"]
            cap = 1000.0 * 1e-9 * 1000.0
            limit = cap / 1e-3 / (9.0 * k)  # a corner's three faces and three films
            films = [(f, 300.0, math.inf, 1e-6) for f in range(6)]
            f, b, _ = _exact_heat(t, 1e-3, k, cap, films, 0.9 * limit, case["steps"], 300.0)
            fields.append(f.reshape(-1))
            books.append(b)
        return {"field": torch.cat(fields), "books": np.array(books)}
    scene = _scene(case, seed)
    d, h = scene["domains"][0], scenes.window(scene)
    if case["domain"] == "block":
        n = case["size"]
        m = scenes.ALUMINIUM_6061
        start = scenes.celsius(d["initial_c"])
        t = torch.full((n, n, n), start, dtype=F64, device="cuda")
        a, b, c = d["hot_spot"]["at"]
        t[c, b, a] = scenes.celsius(d["initial_c"] + d["hot_spot"]["above_k"])
        cap = m["density"] * 1e-9 * m["specific_heat"]
        limit = cap / 1e-3 / (6.0 * m["conductivity"])
        sub = scenes.substeps_for(h, limit)
        first = float(((t - start) * cap).sum())
        f, _, totals = _exact_heat(t, 1e-3, m["conductivity"], cap, [], h / sub, 0, start, per_step=[sub] * case["frames"])
        return {"field": f.reshape(-1), "totals": np.array([first] + totals)}
    n = case["size"]
    dx = 4.4 / (n - 1)
    ny = int(round(3.1 / dx)) + 1
    p = torch.from_numpy(scenes.room_release((n, ny), dx, d["release"])).cuda().reshape(ny, n)
    sub = scenes.substeps_for(h, dx / (scenes.AIR["speed"] * math.sqrt(2.0)))
    f, _, totals = _exact_wave(p, dx, dx * dx, scenes.AIR["density"], scenes.AIR["speed"], h / sub, 0, per_step=[sub] * case["frames"])
    return {"field": f.reshape(-1), "totals": np.array(totals)}
