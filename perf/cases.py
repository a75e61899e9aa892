"""The framework's workloads as timing cases: what a user's program calls, over the sizes and options it is used with.

`listed()` names them, `draw(rng)` gives more of the same ranges, `prepare` / `run` set a case up and take one pass of
it through the public entry points, `work` counts what a pass cannot do without, and `exact` is the same pass in plain
64-bit torch. Vessels are analytic tubes (a straight or bent axis, an optional cosine narrowing), whose signed distance
both sides take as the input; only the voxeliser case and the served stream start from centrelines.
"""
import math

import numpy as np
import torch

from cerebrosim_b200 import batch, lbm, serve, simulate, vessel, wss

DEV = "cuda" if torch.cuda.is_available() else "cpu"

# Steps of a tube taken in `prepare`, so that a pass meets a moving fluid and not the state of rest.
WARM = 100


def listed():
    return [
        # A steady periodic pipe driven by a body force: the smallest vessel in use (a validation run), where the
        # launches and the latency of one step count. One pass = a default chunk of 200 steps.
        {"name": "cylinder", "kind": "steps", "radius": 10.0, "length": 64, "axis": "z", "bend": 0.0, "narrow": 0.0,
         "periodic": True, "model": "regularised", "sigma": 1.0, "tau": 0.8, "storage": "f32", "order": "c",
         "steps": 200},
        # The validation suite's tilted pipe with the solver's defaults (two-relaxation-time collision, C order).
        {"name": "tilted_trt", "kind": "steps", "radius": 10.0, "length": 240, "axis": "tilted", "bend": 0.0,
         "narrow": 0.0, "periodic": False, "model": "trt", "sigma": 1.0, "tau": 0.56, "storage": "f32", "order": "c",
         "steps": 200},
        # The pulsatile pipe of the headline benchmark in single precision and the solver's default node order.
        {"name": "pipe", "kind": "steps", "radius": 24.0, "length": 192, "axis": "z", "bend": 0.0, "narrow": 0.0,
         "periodic": False, "model": "regularised", "sigma": 1.0, "tau": 0.55, "storage": "f32", "order": "c",
         "steps": 200},
        # A bent, stenosed artery of about 1.5 M nodes, in the node order that the tuner picks for such vessels: the
        # production run of one vessel, in FP32 and in the 16-bit storage that keeps its results within 1 %.
        {"name": "artery", "kind": "steps", "radius": 34.0, "length": 440, "axis": "x", "bend": 20.0, "narrow": 0.4,
         "periodic": False, "model": "regularised", "sigma": 1.0, "tau": 0.52, "storage": "f32",
         "order": "axis-boundary-first", "steps": 200},
        {"name": "artery_f16", "kind": "steps", "radius": 34.0, "length": 440, "axis": "x", "bend": 20.0,
         "narrow": 0.4, "periodic": False, "model": "regularised", "sigma": 1.0, "tau": 0.52, "storage": "f16",
         "order": "axis-boundary-first", "steps": 200},
        # A heartbeat of the artery solver: resistance outlets, flows and probes sampled every few steps, coarse
        # frames of the fields, as the production loop records them.
        {"name": "heartbeat", "kind": "beat", "radius": 20.0, "length": 160, "axis": "x", "bend": 6.0, "narrow": 0.3,
         "tau": 0.52, "storage": "f32", "order": "axis-boundary-first", "steps": 400, "every": 20, "frames": 4},
        # A sweep: uneven vessels advanced together in 16-bit storage.
        {"name": "sweep", "kind": "sweep", "count": 6, "nodes_lo": 60000, "nodes_hi": 800000, "tau": 0.52,
         "storage": "f16", "order": "axis-boundary-first", "schedule": "fused", "steps": 200},
        # A vessel's signed distance from its centrelines, the first thing done for each new vessel.
        {"name": "voxelise", "kind": "voxelise", "length": 20.0, "radius": 1.5, "narrow": 0.45, "dx": 0.08},
        # The lattice tables of a voxelised vessel.
        {"name": "tables", "kind": "tables", "radius": 28.0, "length": 360, "axis": "x", "bend": 30.0, "narrow": 0.3},
        # From host tables to fields: a solver built, a short run, the fields read back (a parameter study).
        {"name": "host_to_fields", "kind": "study", "radius": 24.0, "length": 192, "axis": "z", "bend": 0.0,
         "narrow": 0.0, "model": "regularised", "tau": 0.55, "storage": "f32", "order": "boundary-first", "steps": 20},
        # Wall shear stress of one frame at the wall's vertices.
        {"name": "shear", "kind": "shear", "vertices": 150000, "neighbours": 48, "radius": 30.0, "length": 300},
        # Requests served together, built and run as they come off the queue: the whole serving call.
        {"name": "served", "kind": "served", "requests": 4, "nodes_lo": 150000, "nodes_hi": 900000, "beats": 2,
         "storage": "f16", "order": "c", "steps": 1000},
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    """One more case: single vessels half of the time, of 10 thousand to 1.5 million nodes."""
    kind = rng.choice(["steps"] * 6 + ["beat", "sweep", "voxelise", "tables", "study", "shear", "served"])
    order = rng.choice(["c", "c", "axis", "split", "axis-split", "boundary-first", "axis-boundary-first"])
    storage = rng.choice(["f32", "f32", "f16", "f16", "bf16"])
    model = rng.choice(["regularised", "regularised", "regularised", "trt"])
    axis = rng.choice(["x", "z", "tilted"])
    radius = _log(rng, 7.0, 34.0)
    length = int(max(40, radius * rng.uniform(5.0, 12.0)))
    c = {"kind": kind, "radius": round(radius, 3), "length": length, "axis": axis,
         "bend": round(rng.choice([0.0, rng.uniform(0.0, 0.6) * radius]), 3), "narrow": round(rng.uniform(0, 0.5), 3)}
    if kind == "steps":
        periodic = rng.random() < 0.2
        if periodic:
            c.update(axis="z", bend=0.0, narrow=0.0)
        return dict(c, periodic=periodic, model=model, sigma=rng.choice([1.0, 1.0, 1.0, 0.6]),
                    tau=round(rng.uniform(0.52, 0.8), 3), storage=storage, order=order,
                    steps=rng.choice([1, 20, 100, 200, 200, 201]))
    if kind == "beat":
        every = rng.choice([10, 20, 40])
        c.update(axis="x", radius=min(c["radius"], 24.0), length=min(length, 200))
        return dict(c, tau=0.52, storage=rng.choice(["f32", "f16"]), order=order, steps=400, every=every, frames=2)
    if kind == "sweep":
        lo = _log(rng, 20000, 200000)
        return {"kind": kind, "count": rng.randint(2, 8), "nodes_lo": int(lo), "nodes_hi": int(lo * rng.uniform(1, 4)),
                "tau": 0.52, "storage": storage, "order": order,
                "schedule": rng.choice(["fused", "by-instance", "concurrent:2"]), "steps": 100}
    if kind == "voxelise":
        return {"kind": kind, "length": round(rng.uniform(12.0, 24.0), 2), "radius": round(rng.uniform(1.0, 2.0), 3),
                "narrow": round(rng.uniform(0.0, 0.6), 3), "dx": round(_log(rng, 0.07, 0.25), 4)}
    if kind == "tables":
        return c
    if kind == "study":
        c.update(radius=min(c["radius"], 24.0), length=min(length, 240))
        return dict(c, model=model, tau=round(rng.uniform(0.52, 0.7), 3), storage=storage, order=order,
                    steps=rng.choice([1, 5, 20, 50]))
    if kind == "shear":
        return {"kind": kind, "vertices": int(_log(rng, 3000, 200000)), "neighbours": rng.choice([12, 24, 48, 48]),
                "radius": round(rng.uniform(12.0, 30.0), 2), "length": rng.randint(60, 300)}
    lo = _log(rng, 80000, 160000)
    return {"kind": kind, "requests": rng.randint(1, 4), "nodes_lo": int(lo), "nodes_hi": int(2.5 * lo),
            "beats": rng.randint(1, 2), "storage": rng.choice(["f16", "f32"]), "order": order, "steps": 1000}


# ---- vessels --------------------------------------------------------------------------------------------------------
AXES = {"x": (1.0, 0.0, 0.0), "z": (0.0, 0.0, 1.0), "tilted": (1 / 3, 2 / 3, 2 / 3)}


def tube(case, seed):
    """Signed distance (float32 on the device, negative inside) and openings of a case's tube. The seed stretches the
    distance from place to place: it moves the wall within its cells and leaves the set of fluid cells alone."""
    rng = np.random.default_rng([seed, 1])
    R, L, narrow = float(case["radius"]), int(case["length"]), float(case.get("narrow", 0.0))
    shift = (0.31, 0.17, 0.5)
    wave, phase = rng.uniform(0.05, 0.3, size=3), rng.uniform(0, 2 * math.pi)
    f64 = {"dtype": torch.float64, "device": DEV}
    if case.get("periodic"):
        n = int(math.ceil(2 * R)) + 5
        x = torch.arange(n, **f64) - (n / 2 - 0.5)
        r = torch.hypot(x[:, None] - shift[0], x[None, :] - shift[1])
        r = (r - R) * (1 + 0.2 * torch.sin(wave[0] * x[:, None] + wave[1] * x[None, :] + phase))
        return r.to(torch.float32)[:, :, None].expand(n, n, L).contiguous(), []
    ax = np.array(AXES[case["axis"]])
    side = np.cross(ax, [0.0, 1.0, 0.0] if abs(ax[1]) < 0.9 else [1.0, 0.0, 0.0])
    side /= np.linalg.norm(side)
    bend = float(case.get("bend", 0.0))
    reach = R * np.sqrt(np.clip(1 - ax ** 2, 0, 1)) + bend * np.abs(side) + 3
    lo, hi = np.minimum(0, ax * L) - reach, np.maximum(0, ax * L) + reach
    dims = np.ceil(hi - lo).astype(int) + 1
    start = -lo + np.array(shift)
    g = [torch.arange(int(d), **f64) - float(o) for d, o in zip(dims, start)]
    g = [g[0][:, None, None], g[1][None, :, None], g[2][None, None, :]]
    s = sum(g[a] * float(ax[a]) for a in range(3))
    off = bend * torch.sin(2 * math.pi * s / L)
    rad = torch.sqrt(sum((g[a] - s * float(ax[a]) - off * float(side[a])) ** 2 for a in range(3)))
    w = torch.where((s / L - 0.5).abs() < 0.1, 0.5 + 0.5 * torch.cos(10 * math.pi * (s / L - 0.5)), 0.0)
    phi = torch.maximum(torch.maximum(rad - R * (1 - narrow * w), -s), s - L)
    phi = phi * (1 + 0.2 * torch.sin(sum(g[a] * float(wave[a]) for a in range(3)) + phase))
    return phi.to(torch.float32), [{"kind": "inlet", "centre": start, "normal": -ax, "radius": R},
                 {"kind": "outlet", "centre": start + ax * L, "normal": ax, "radius": R}]


def nodes(case):
    """Fluid nodes of a case's tube, from its volume."""
    full = math.pi * case["radius"] ** 2 * case["length"]
    return full * (1 - 0.2 * case.get("narrow", 0.0))


def drive(seed, mean):
    """Fourier coefficients of a pulsatile inflow."""
    rng = np.random.default_rng([seed, 2])
    a = 0.25 * mean * rng.uniform(-1, 1, size=(3, 2)) / np.arange(1, 4)[:, None]
    return [mean] + a.ravel().tolist()


PERIOD = 2000
FORCE = (0.0, 0.0, 1e-6)


def settings(s, case, seed):
    """Drive, outlets, force and sponge of a vessel, as a user's program sets them."""
    if case.get("periodic"):
        s.set_force(FORCE)
        s.set_drive(drive(seed, 1.0), period=PERIOD)
        return s
    s.set_sponge(8, 0.6)
    s.set_outlet_pressure([0.001])
    s.set_drive(drive(seed, 0.03), period=PERIOD, ramp=WARM)
    return s


def now(s):
    """Density deviation and velocity per cell, in the lattice's order, on the device."""
    rho, u = s.rho, s.vels[s.cur]
    return {"rho": rho, "u": u} if s.inv is None else {"rho": rho[s.inv], "u": u[s.inv]}


def member_cases(case):
    """The vessels of a sweep: tubes six radii long, sizes evenly spread over the logarithm."""
    out = []
    for k in range(case["count"]):
        n = case["nodes_lo"] * (case["nodes_hi"] / case["nodes_lo"]) ** (k / max(1, case["count"] - 1))
        r = (n / (6 * math.pi)) ** (1 / 3)
        out.append({"radius": r, "length": int(6 * r), "axis": "xz"[k % 2], "bend": 0.3 * r, "narrow": 0.1 * (k % 5),
                    "tau": case["tau"]})
    return out


def centrelines(case, seed):
    """A parent on a bent axis (the seed's) with a cosine narrowing and a straight side branch, in mm, in the geometry
    format the voxeliser takes."""
    rng = np.random.default_rng([seed, 3])
    L, R = case["length"], case["radius"]
    x = np.linspace(0.0, L, int(L / 0.1) + 1)
    amp = rng.uniform(0.3, 1.0, size=4)
    C = np.column_stack([x, amp[0] * np.sin(3 * x / L) + amp[1] * np.sin(5 * x / L),
                         amp[2] * np.sin(4 * x / L) + amp[3] * np.cos(5 * x / L)])
    w = np.where(np.abs(x - L / 2) < 1.5, 0.5 + 0.5 * np.cos(2 * math.pi * (x - L / 2) / 3.0), 0.0)
    radius = R * (1 - case["narrow"] * w)

    def unit(v):
        return v / np.linalg.norm(v)
    d = np.array([math.cos(0.7), math.sin(0.7), 0.0])
    B = C[int(0.7 * len(x))] + np.linspace(0.0, 0.6 * L, int(6 * L))[:, None] * d
    return {"branches": {
        "trunk": {"C": C, "R0": np.full(len(x), R), "R": radius,
                  "caps": {"start": (C[0], -unit(C[1] - C[0])), "end": (C[-1], unit(C[-1] - C[-2]))}},
        "branch": {"C": B, "R0": np.full(len(B), 0.65 * R), "R": np.full(len(B), 0.65 * R),
                   "caps": {"start": None, "end": (B[-1], d)}}}}


def voxel_box(case):
    """The box that holds any seed's vessel of a voxeliser case, half a millimetre around it."""
    L, r = case["length"], case["radius"] + 0.5
    return np.array([-r, -2 - r, -2 - r]), np.array([0.7 * L + 0.6 * L * math.cos(0.7) + r,
                                                     2 + 0.6 * L * math.sin(0.7) + r, 2 + r])


def voxel_shape(case):
    lo, hi = voxel_box(case)
    return tuple(int(n) for n in np.ceil((hi - lo) / case["dx"]).astype(int) + 1)


def wall_cells(case, seed):
    """Vertices on a cylinder's wall with their inward normals, and for each the cells of the box around the point
    just inside it, with fit coefficients; velocities of a developed flow with a seeded disturbance."""
    V, K, R, L = case["vertices"], case["neighbours"], case["radius"], case["length"]
    gen = torch.Generator().manual_seed(seed)
    n = int(2 * R) + 5
    x = torch.arange(n, dtype=torch.float64) - (n - 1) / 2
    rr = torch.hypot(x[:, None], x[None, :])
    inside = rr < R
    plane = int(inside.sum())
    rank = torch.full((n, n), -1, dtype=torch.int64)
    rank[inside] = torch.arange(plane)
    # vertices walk along the wall ring by ring, as a surface mesh numbers them
    th = torch.arange(V, dtype=torch.float64) * (2 * math.pi / max(8.0, 2 * math.pi * R))
    z = torch.arange(V, dtype=torch.float64) * ((L - 8) / V) + 4
    nrm = -torch.stack([torch.cos(th), torch.sin(th), torch.zeros_like(th)], 1)
    base = -nrm[:, :2] * (R - 2.0) + (n - 1) / 2
    i0, j0, k0 = (base[:, 0].round().long(), base[:, 1].round().long(), z.long())
    off = torch.tensor([(a, b, c) for c in (0, 1, -1) for a in range(-2, 2) for b in range(-2, 2)])[:K]
    cell = rank[(i0[:, None] + off[:, 0]).clamp(0, n - 1), (j0[:, None] + off[:, 1]).clamp(0, n - 1)]
    idx = torch.where(cell >= 0, (k0[:, None] + off[:, 2]) * plane + cell.clamp(min=0), 0)
    c = torch.where(cell >= 0, torch.randn(V, K, generator=gen, dtype=torch.float64), 0.0)
    u = torch.zeros(L, plane, 3)
    u[:, :, 2] = (0.3 * (1 - (rr[inside] / R) ** 2)).to(torch.float32)
    u += 0.02 * torch.randn(L, plane, 3, generator=gen)
    return nrm.to(torch.float32), idx.to(torch.int32), c.to(torch.float32), u.reshape(-1, 3)


def requests(case, seed):
    """Uneven vessels asked for together, each at a mean pressure of its own."""
    rng = np.random.default_rng([seed, 4])
    n = case["requests"]
    sizes = case["nodes_lo"] * (case["nodes_hi"] / case["nodes_lo"]) ** (np.arange(n) / max(1, n - 1))
    return [{"id": k, "arrival": 0.1 * k, "seed": 1000 + k, "stenosis": 0.9 * ((k * 0.37 + 0.2) % 1.0),
             "pressure": float(rng.uniform(70, 145)), "beats": 1 + k % case["beats"], "nodes": float(sizes[k])}
            for k in range(n)]


# ---- a pass ---------------------------------------------------------------------------------------------------------
def solver(case, seed, lat, **kw):
    return settings(lbm.Solver(lat, (case["tau"] - 0.5) / 3.0, model=case.get("model", "regularised"),
                               sigma=case.get("sigma", 1.0), storage=case["storage"], order=case["order"], **kw),
                    case, seed)


def tube_lattice(case, seed, host=False):
    phi, ops = tube(case, seed)
    return lbm.build_lattice(phi, [0.0, 0.0, 0.0], 1.0, openings=ops, periodic=(2,) if case.get("periodic") else (),
                             host=host)


def open_ends(case, seed):
    """The heartbeat's tube with both ends as pressure boundaries: end 0 follows the drive."""
    phi, ops = tube(case, seed)
    return phi, [dict(o, kind="outlet") for o in ops]


PREF, ALPHA, RESIST = 0.002, 0.01, (0.0, 4e-5)


def beat_flux(coords, ends):
    """The flow slabs of the heartbeat's ends, 6 to 10 cells inside each."""
    return simulate.flux_slabs({"origin": np.zeros(3), "coords": coords}, ends, 1.0, slab_mm=(6.0, 10.0))


def probe_cells(coords, case):
    """Probes: balls of cells in six planes along the vessel."""
    x = coords[:, 0]
    idx, slot = [], []
    for k in range(6):
        m = np.flatnonzero(np.abs(x - (x.min() + (k + 0.5) * (x.max() - x.min()) / 6)) < 2)
        idx.append(m)
        slot.append(np.full(len(m), k))
    return np.concatenate(idx), np.concatenate(slot)


def prepare(case, seed):
    kind = case["kind"]
    if kind == "steps":
        s = solver(case, seed, tube_lattice(case, seed))
        s.run(WARM)
        return {"kind": kind, "s": s, "steps": case["steps"], "periodic": case["periodic"]}
    if kind == "beat":
        phi, ends = open_ends(case, seed)
        lat = lbm.build_lattice(phi, [0.0, 0.0, 0.0], 1.0, openings=ends)
        s = simulate.ArterySolver(lat, (case["tau"] - 0.5) / 3.0, beat_flux(lat["coords"], ends), RESIST, PREF, ALPHA,
                                  model="regularised", storage=case["storage"], order=case["order"])
        s.set_sponge(8, 0.6, kinds=("outlet",))
        s.set_outlet_pressure([0.0, -PREF])
        s.set_drive(drive(seed, 0.003), period=case["steps"], ramp=case["steps"] // 2)
        probes = simulate.Probes(s, *probe_cells(lat["coords"], case), 6)
        cmap = simulate.CoarseMap(s, lat, 0.05)
        return {"kind": kind, "s": s, "case": case, "probes": probes, "cmap": cmap}
    if kind == "sweep":
        sols = [solver(dict(c, storage=case["storage"], order=case["order"]), seed + 31 * k,
                       tube_lattice(c, seed + 31 * k)) for k, c in enumerate(member_cases(case))]
        b = batch.BatchSolver(sols, schedule=case["schedule"])
        b.run(WARM)
        return {"kind": kind, "b": b, "steps": case["steps"]}
    if kind == "voxelise":
        return {"kind": kind, "g": centrelines(case, seed), "dx": case["dx"], "box": voxel_box(case)}
    if kind == "tables":
        phi, ops = tube(case, seed)
        return {"kind": kind, "phi": phi, "openings": ops}
    if kind == "study":
        lat = dict(tube_lattice(case, seed, host=True))
        lat.pop("_dev")
        for k in ("nbr", "q", "uin"):
            lat[k] = torch.from_numpy(np.ascontiguousarray(lat[k])).pin_memory()
        return {"kind": kind, "lat": lat, "case": case, "seed": seed}
    if kind == "shear":
        nrm, idx, c, u = wall_cells(case, seed)
        return {"kind": kind, "shear": wss.Shear(nrm.numpy(), idx.numpy(), c.numpy(), len(u)), "u": u.cuda()}
    return {"kind": kind, "case": case, "specs": requests(case, seed)}


def run(state):
    kind = state["kind"]
    if kind == "steps":
        state["s"].run(state["steps"])
        out = now(state["s"])
        if state["periodic"]:          # nothing drives a pressure there: the density is 1 and its deviation rounding
            out["rho"] = 1.0 + out["rho"]
        return out
    if kind == "beat":
        s, c = state["s"], state["case"]
        series, frames = simulate.run_beats(s, c["steps"], s.steps // c["steps"] + 1, c["every"], state["probes"],
                                            state["cmap"], frames=c["frames"])
        return {"series": series, "frames": {"p": frames["p"], "u": frames["u"]}, **now(s)}
    if kind == "sweep":
        state["b"].run(state["steps"])
        return [now(s) for s in state["b"].members]
    if kind == "voxelise":
        return vessel.sdf_grid(state["g"], state["dx"], *state["box"], host=False)[0]
    if kind == "tables":
        lat = lbm.build_lattice(state["phi"], [0.0, 0.0, 0.0], 1.0, openings=state["openings"], host=False)
        return {**{k: lat["_dev"][k] for k in ("nbr", "q", "uin", "coords")}, "counts": [
            lat["counts"]["wall"], lat["counts"]["inlet"], *lat["counts"]["outlet"]]}
    if kind == "study":
        s = solver(state["case"], state["seed"], state["lat"])
        s.run(state["case"]["steps"])
        p, u = s.fields()
        return {"p": p, "u": u}
    if kind == "shear":
        return state["shear"](state["u"])
    c = state["case"]
    server = serve.Server(storage=c["storage"], order=c["order"], steps_per_beat=c["steps"], chunk=c["steps"])
    done = server.serve(state["specs"], realtime=False)
    return [{"p": r.fields[0], "u": r.fields[1]} for r in done]


def work(case):
    """Bytes and flops of a pass. A step reads and writes each node's 27 populations and its velocity (the Galilean
    differences) and some 400 flops; the density is written once a pass."""
    kind = case["kind"]
    if kind in ("steps", "beat", "sweep", "study", "served"):
        size = 4 if case["storage"] == "f32" else 2
        if kind == "sweep":
            n = sum(nodes(c) for c in member_cases(case))
            steps = n * case["steps"]
        elif kind == "served":
            r = requests(case, 0)
            n = sum(x["nodes"] for x in r)
            steps = sum(x["nodes"] * x["beats"] for x in r) * case["steps"]
        else:
            n = nodes(case)
            steps = n * case["steps"]
        tables = n * (27 * 8 + 12) if kind == "study" else 0
        return {"bytes": steps * (54 * size + 24) + 4 * n + tables, "flops": 400 * steps}
    if kind == "voxelise":
        voxels = float(np.prod(voxel_shape(case)))
        return {"bytes": 4 * voxels, "flops": 100 * voxels}
    if kind == "tables":
        n = nodes(case)
        box = case["length"] * (2 * case["radius"] + 6) * (2 * (case["radius"] + case["bend"]) + 6)
        return {"bytes": 4 * box + n * (27 * 8 + 24), "flops": 27 * n}
    v, k = case["vertices"], case["neighbours"]
    cells = math.pi * case["radius"] ** 2 * case["length"]
    return {"bytes": 8 * v * k + 24 * v + 12 * min(cells, v * k), "flops": 14 * v * k}


# ---- the same in 64 bits --------------------------------------------------------------------------------------------
C = torch.tensor([[0, 0, 0], [1, 0, 0], [-1, 0, 0], [0, 1, 0], [0, -1, 0], [0, 0, 1], [0, 0, -1], [1, 1, 0],
                  [-1, -1, 0], [1, -1, 0], [-1, 1, 0], [1, 0, 1], [-1, 0, -1], [1, 0, -1], [-1, 0, 1], [0, 1, 1],
                  [0, -1, -1], [0, 1, -1], [0, -1, 1], [1, 1, 1], [-1, -1, -1], [1, 1, -1], [-1, -1, 1], [1, -1, 1],
                  [-1, 1, -1], [-1, 1, 1], [1, -1, -1]])
W = torch.tensor([8 / 27] + [2 / 27] * 6 + [1 / 54] * 12 + [1 / 216] * 8, dtype=torch.float64)
OPP = torch.tensor([0] + [i + 1 if i % 2 else i - 1 for i in range(1, 27)])


def plain_lattice(phi, openings, periodic=()):
    """Pull sources (>= 0 node, -1 wall, -2 inlet, -3 - k outlet k), wall fractions, inlet profile and coordinates."""
    d = phi.device
    dims = torch.tensor(phi.shape, device=d)
    fluid = phi < 0
    coords = fluid.nonzero()
    n = len(coords)
    rank = torch.full(phi.shape, -1, dtype=torch.int64, device=d)
    rank[fluid] = torch.arange(n, device=d)
    nbr = torch.empty((27, n), dtype=torch.int64, device=d)
    q = torch.full((27, n), 0.5, dtype=torch.float64, device=d)
    here = phi[fluid].double()
    order = [o for o in openings if o["kind"] == "inlet"] + [o for o in openings if o["kind"] == "outlet"]

    def place(o, p):
        c, m = (torch.as_tensor(np.asarray(o[k], float), device=d) for k in ("centre", "normal"))
        rel = p - c
        along = rel @ m
        return along, torch.linalg.norm(rel - along[:, None] * m, dim=1)
    for i in range(27):
        x = coords - C[i].to(d)
        for a in periodic:
            x[:, a] %= dims[a]
        ok = ((x >= 0) & (x < dims)).all(1)
        y = torch.minimum(x.clamp(min=0), dims - 1)
        src = torch.where(ok, rank[y[:, 0], y[:, 1], y[:, 2]], -1)
        miss = (src < 0).nonzero().flatten()
        code = torch.full_like(miss, -1)
        k = 0
        for o in order:
            along, across = place(o, x[miss].double())
            hit = (code == -1) & (along >= -1e-6) & (across < o["radius"] + 1.0)
            code[hit] = -2 if o["kind"] == "inlet" else -3 - k
            k += o["kind"] == "outlet"
        src[miss] = code
        f = -here[miss] / (phi[y[miss, 0], y[miss, 1], y[miss, 2]].double() - here[miss])
        f = torch.where(ok[miss] & torch.isfinite(f), f.clamp(1e-3, 1.0), 0.5)
        q[i, miss] = torch.where(code == -1, f, 0.5)
        nbr[i] = src
    uin = torch.zeros((n, 3), dtype=torch.float64, device=d)
    inlets = [o for o in order if o["kind"] == "inlet"]
    if inlets:
        o = inlets[-1]
        prof = 2.0 * (1.0 - (place(o, coords.double())[1] / o["radius"]) ** 2).clamp(min=0)
        cell = (nbr == -2).any(0)
        uin[cell] = -prof[cell, None] * torch.as_tensor(np.asarray(o["normal"], float), device=d)
    return {"nbr": nbr, "q": q, "uin": uin, "coords": coords}


def third(c, u):
    x, y, z = u
    cx, cy, cz = (float(v) for v in c)
    a, b, e = cx * cx - 1 / 3, cy * cy - 1 / 3, cz * cz - 1 / 3
    return 13.5 * (a * (cy * x * x * y + cz * x * x * z) + b * (cx * x * y * y + cz * y * y * z)
                   + e * (cx * x * z * z + cy * y * z * z)) + 27.0 * cx * cy * cz * x * y * z


class Plain:
    """The scheme in 64-bit torch: pull, boundary links, collision, and the resistance outlets when a flux is given."""

    def __init__(self, lat, tau, model, sigma, coef, period, ramp, force=(0.0, 0.0, 0.0), sponge=(), p_out=(0.0,),
                 flux=None):
        self.d = d = lat["nbr"].device
        self.lat, self.model, self.sigma, self.flux = lat, model, sigma, flux
        self.coef, self.period, self.ramp, self.tick = np.float32(coef).astype(float), period, ramp, 0
        self.force = [float(np.float32(x)) for x in force]
        nbr = lat["nbr"]
        self.n = n = nbr.shape[1]
        self.src = nbr.clamp(min=0)
        io = OPP.to(d)
        self.links = []
        for i in range(27):
            at = (nbr[i] < 0).nonzero().flatten()
            self.links.append((at, nbr[i, at], lat["q"][i, at], nbr[io[i], at]))
        t = torch.full((n,), float(tau), dtype=torch.float64, device=d)
        for o in sponge:
            c, m = (torch.as_tensor(np.asarray(o[k], float), device=d) for k in ("centre", "normal"))
            rel = lat["coords"].double() - c
            along = rel @ m
            near = torch.linalg.norm(rel - along[:, None] * m, dim=1) < 1.5 * o["radius"]
            w = (1.0 + along / 8.0).clamp(0, 1)
            t = torch.maximum(t, torch.where(near, tau + (0.6 - tau) * w * w * (3 - 2 * w), t))
        self.om = 1.0 / t
        self.inlet = (nbr == -2).any(0)
        z = {"dtype": torch.float64, "device": d}
        self.f, self.u, self.rho = torch.zeros((27, n), **z), torch.zeros((3, n), **z), torch.zeros(n, **z)
        self.p_out = [float(np.float32(p)) for p in p_out]
        self.q_last = [0.0] * len(self.p_out)

    def value(self):
        ph = 2 * math.pi * (self.tick % self.period) / self.period
        v = self.coef[0] + sum(self.coef[2 * k - 1] * math.cos(k * ph) + self.coef[2 * k] * math.sin(k * ph)
                               for k in range(1, (len(self.coef) + 1) // 2))
        return v * (0.5 - 0.5 * math.cos(math.pi * self.tick / self.ramp)) if self.tick < self.ramp else v

    def slope(self, a):
        """Central difference of the velocity along axis a, with walls at their distance and openings flat."""
        h, v = [], []
        for i in (1 + 2 * a, 2 + 2 * a):
            s = self.lat["nbr"][i]
            wall = s == -1
            h.append(torch.where(wall, self.lat["q"][i].clamp(min=0.1), 1.0))
            v.append(torch.where(wall, 0.0, torch.where(s >= 0, self.u[:, s.clamp(min=0)], self.u)))
        h1, h2 = h
        return (h1 * h1 * (v[1] - self.u) + h2 * h2 * (self.u - v[0])) / (h1 * h2 * (h1 + h2))

    def step(self):
        dv, f0, uin = self.value(), self.f, self.lat["uin"].T
        f = torch.gather(f0, 1, self.src)
        for i, (at, code, q, second) in enumerate(self.links):
            io, w, c = int(OPP[i]), float(W[i]), C[i].tolist()
            fo = f0[io, at]
            far = torch.where(second >= 0, 2 * q * fo + (1 - 2 * q) * f0[io, second.clamp(min=0)], fo)
            v = torch.where(q < 0.5, far, fo / (2 * q) + (2 * q - 1) / (2 * q) * f0[i, at])
            ci = sum(c[a] * uin[a, at] for a in range(3)) * dv
            v = torch.where(code == -2, fo + 6 * w * ci, v)
            up = self.u[:, at]
            cu = sum(c[a] * up[a] for a in range(3))
            for k, p in enumerate(self.p_out):
                v = torch.where(code == -3 - k, -fo + 2 * w * (3 * p + 4.5 * cu * cu - 1.5 * (up * up).sum(0)), v)
            f[i, at] = v
        om, c64 = self.om, C.to(self.d).double()
        dr = f.sum(0)
        F = [x * dv for x in self.force]
        u = torch.stack([(c64[:, a] @ f) + 0.5 * F[a] for a in range(3)])
        usq, uF = (u * u).sum(0), sum(u[a] * F[a] for a in range(3))
        G = [self.slope(a) for a in range(3)]
        ed = [3.0 / om * u[a] * u[a] * G[a][a] for a in range(3)]
        ut = uin * dv
        out = torch.empty_like(f)
        if self.model == "regularised":
            P = {}
            cus = [sum(c * u[a] for a, c in enumerate(C[i].tolist())) for i in range(27)]
            neq = [f[i] - float(W[i]) * (dr + 3 * cus[i] + 4.5 * cus[i] ** 2 - 1.5 * usq) for i in range(27)]
            for a in range(3):
                for b in range(a, 3):
                    p = sum(float(C[i, a] * C[i, b]) * neq[i] for i in range(27) if C[i, a] * C[i, b])
                    if self.sigma < 1:
                        p = self.sigma * p - (1 - self.sigma) / (3 * om) * (G[a][b] + G[b][a])
                    P[a, b] = P[b, a] = p - ed[a] if a == b else p
            tr = (P[0, 0] + P[1, 1] + P[2, 2]) / 3
            for i in range(27):
                c, w, cu = C[i].tolist(), float(W[i]), cus[i]
                cF = sum(c[a] * F[a] for a in range(3))
                quad = sum(c[a] * c[b] * P[a, b] for a in range(3) for b in range(3))
                out[i] = (w * (dr + 3 * cu + 4.5 * cu * cu - 1.5 * usq + third(c, u))
                          + (1 - om) * w * (4.5 * (quad - tr) - 1.5 * cF)
                          + (1 - 0.5 * om) * w * (3 * cF + 9 * cu * cF - 3 * uF))
        else:
            om_m = 1.0 / (0.5 + 0.1875 / (1.0 / om - 0.5))
            dd = [-(1 - om) * e for e in ed]
            tr = (dd[0] + dd[1] + dd[2]) / 3
            for i in range(27):
                c, w = C[i].tolist(), float(W[i])
                cv, cF = sum(c[a] * u[a] for a in range(3)), sum(c[a] * F[a] for a in range(3))
                other = f[int(OPP[i])]
                out[i] = (f[i] - om * (0.5 * (f[i] + other) - w * (dr + 4.5 * cv * cv - 1.5 * usq))
                          - om_m * (0.5 * (f[i] - other) - w * (3 * cv + third(c, u)))
                          + (1 - 0.5 * om) * w * (9 * cv * cF - 3 * uF) + (1 - 0.5 * om_m) * w * 3 * cF
                          + w * 4.5 * (sum(c[a] * c[a] * dd[a] for a in range(3)) - tr))
        if bool(self.inlet.any()):
            m = self.inlet
            t = ut[:, m]
            for i in range(27):
                c, w = C[i].tolist(), float(W[i])
                cu = sum(c[a] * t[a] for a in range(3))
                out[i, m] = w * (dr[m] + 3 * cu + 4.5 * cu * cu - 1.5 * (t * t).sum(0) + third(c, t))
            u[:, m] = t
        self.f, self.u, self.rho = out, u, dr
        self.tick += 1
        if self.flux is not None:
            flow = (u[:, self.flux["idx"]] * self.flux["w"].T).sum(0)
            self.q_last = [float(flow[self.flux["slot"] == k].sum()) for k in range(len(self.p_out))]
            self.p_out = [dv] + [self.p_out[k] + ALPHA * (float(np.float32(RESIST[k])) * self.q_last[k] - PREF
                                                         - self.p_out[k]) for k in range(1, len(self.p_out))]

    def run(self, steps):
        for _ in range(steps):
            self.step()
        return self


def plain_tube(case, seed):
    """The 64-bit run of a tube with the settings that `settings` makes."""
    phi, ops = tube(case, seed)
    periodic = bool(case.get("periodic"))
    lat = plain_lattice(phi, ops, (2,) if periodic else ())
    model, sigma = case.get("model", "regularised"), case.get("sigma", 1.0)
    if periodic:
        return Plain(lat, case["tau"], model, sigma, drive(seed, 1.0), PERIOD, 0, force=FORCE)
    return Plain(lat, case["tau"], model, sigma, drive(seed, 0.03), PERIOD, WARM, sponge=ops, p_out=(0.001,))


def plain_beat(case, seed):
    phi, ends = open_ends(case, seed)
    lat = plain_lattice(phi, ends)
    d = phi.device
    coords = lat["coords"].cpu().numpy()
    thick, idx, w, slot = 4.0, [], [], []
    for k, e in enumerate(ends):
        rel = coords - e["centre"]
        depth = -(rel @ e["normal"])
        near = np.linalg.norm(rel + depth[:, None] * e["normal"], axis=1) < 1.3 * e["radius"]
        m = np.flatnonzero(near & (depth >= 6.0) & (depth < 10.0))
        idx.append(m)
        slot.append(np.full(len(m), k))
        w.append(np.tile((-1.0 if k == 0 else 1.0) * e["normal"] / thick, (len(m), 1)))
    flux = {"idx": torch.as_tensor(np.concatenate(idx), device=d), "slot": torch.as_tensor(np.concatenate(slot), device=d),
            "w": torch.as_tensor(np.vstack(w), device=d)}
    s = Plain(lat, case["tau"], "regularised", 1.0, drive(seed, 0.003), case["steps"], case["steps"] // 2, sponge=ends,
              p_out=(0.0, -PREF), flux=flux)
    cells, slots = (torch.as_tensor(x, device=d) for x in probe_cells(coords, case))
    per = torch.bincount(slots, minlength=6).double()
    _, inv = np.unique(coords // 2, axis=0, return_inverse=True)
    inv = torch.as_tensor(inv.ravel(), device=d)
    size = torch.bincount(inv).double()
    series = {"step": None, "Q": [], "p_open": [], "p_probe": [], "umax": []}
    frames = {"p": [], "u": []}
    for k in range(1, case["steps"] // case["every"] + 1):
        s.run(case["every"])
        series["Q"].append(s.q_last)
        series["p_open"].append(s.p_out)
        series["p_probe"].append((torch.bincount(slots, s.rho[cells] / 3, 6) / per).tolist())
        series["umax"].append(float(torch.linalg.norm(s.u[:, cells], dim=0).max()))
        if (k * case["every"]) % (case["steps"] // case["frames"]) == 0:
            frames["p"].append((torch.bincount(inv, s.rho / 3) / size).cpu().numpy())
            frames["u"].append(np.stack([(torch.bincount(inv, s.u[a]) / size).cpu().numpy() for a in range(3)], 1))
    return {"series": {k: None if v is None else np.array(v) for k, v in series.items()},
            "frames": {k: np.array(v) for k, v in frames.items()}, "rho": s.rho, "u": s.u.T}


def plain_distance(case, seed):
    """Round cones, flat caps and a smooth union on the voxel grid, a slab of voxels at a time."""
    g = centrelines(case, seed)
    shape, lo = voxel_shape(case), voxel_box(case)[0]
    f64 = {"dtype": torch.float64, "device": DEV}
    out = torch.empty(shape, **f64)
    ax = [torch.arange(n, **f64) * case["dx"] + float(o) for n, o in zip(shape, lo)]
    for i in range(shape[0]):
        p = torch.stack([ax[0][i].expand(shape[1], shape[2]), ax[1][:, None].expand(shape[1], shape[2]),
                         ax[2][None, :].expand(shape[1], shape[2])], -1)
        d = torch.full(shape[1:], 1e9, **f64)
        for b in g["branches"].values():
            P, R = torch.as_tensor(b["C"], **f64), torch.as_tensor(b["R"], **f64)
            db = torch.full(shape[1:], 1e9, **f64)
            for k in range(0, len(P) - 1, 64):
                A, B = P[k:min(k + 64, len(P) - 1)], P[k + 1:k + 65]
                ab, r0, r1 = B - A, R[k:k + len(A)], R[k + 1:k + 1 + len(A)]
                rel = p[:, :, None, :] - A
                t = ((rel * ab).sum(-1) / (ab * ab).sum(-1).clamp(min=1e-12)).clamp(0, 1)
                dist = torch.linalg.norm(rel - t[..., None] * ab, dim=-1) - (r0 + (r1 - r0) * t)
                db = torch.minimum(db, dist.min(-1).values)
            for key, r in (("start", float(b["R"][0])), ("end", float(b["R"][-1]))):
                cap = b["caps"][key]
                if cap is not None:
                    rel = p - torch.as_tensor(cap[0], **f64)
                    cut = torch.maximum(db, rel @ torch.as_tensor(cap[1], **f64))
                    db = torch.where(torch.linalg.norm(rel, dim=-1) < 2.5 * r, cut, db)
            h = (0.5 + 0.5 * (db - d) / 0.6).clamp(0, 1)
            d = db + (d - db) * h - 0.6 * h * (1 - h)
        out[i] = d
    return out


def exact(case, seed):
    kind = case["kind"]
    if kind == "steps":
        s = plain_tube(case, seed).run(WARM + case["steps"])
        return {"rho": 1.0 + s.rho if case["periodic"] else s.rho, "u": s.u.T}
    if kind == "beat":
        return plain_beat(case, seed)
    if kind == "sweep":
        out = []
        for k, c in enumerate(member_cases(case)):
            s = plain_tube(c, seed + 31 * k).run(WARM + case["steps"])
            out.append({"rho": s.rho, "u": s.u.T})
        return out
    if kind == "voxelise":
        return plain_distance(case, seed)
    if kind == "tables":
        lat = plain_lattice(*tube(case, seed))
        return {"nbr": None, "q": lat["q"], "uin": lat["uin"], "coords": None, "counts": None}
    if kind == "study":
        s = plain_tube(case, seed).run(case["steps"])
        return {"p": (s.rho / 3).cpu().numpy(), "u": s.u.T.cpu().numpy()}
    if kind == "shear":
        nrm, idx, c, u = (t.to(DEV) for t in wall_cells(case, seed))
        nrm, c, uj = nrm.double(), c.double(), u.double()[idx.long()]
        ut = uj - (uj * nrm[:, None, :]).sum(-1, keepdim=True) * nrm[:, None, :]
        return 0.0035 * 1e3 * (c[..., None] * ut).sum(1)
    return None                # the served vessels are the framework's own generator's
