"""Performance cases of the cloth step: what programs that use this package have it do.

Every case is one pass of such a program through the public API (Simulation,
SpringyMesh, Cloth, Surrogate) over inputs made from a seed.  The physical
parameters are those of feriphys_gb300.workloads (strut constants, vertex
mass, wind, the plane and sphere colliders); the step is 1/30000 s, the step
the learned surrogate's fine solver runs at, so a state that is stepped again
and again stays on a physical trajectory.

kinds
  cloth    one Cloth::new grid: `steps` steps, then the state is read back
           read = "points"    Stateful rows into a fresh host array
                  "vertices"  positions into a fresh host array
                  "pinned"    positions into a pinned host array
                  "export"    render vertices into device memory
                  "exchange"  set_points, the steps, get_points (both pinned)
           woven = True: built as the large benchmark cloth is, from a triangle
           list with noisy rest positions and per-strut stiffness, with a sphere
           under it
  tube     a closed tube (a sleeve): no Cloth::new grid, so the general gather
  batch    many uneven cloths in one simulation, every one with its own wind
  coarse   learned-surrogate rollout with the energy and strain checks on
  train    surrogate training on transitions recorded from the simulation
"""
import math

import numpy as np
import torch

import feriphys_gb300 as fgb

DT = float(np.float32(1.0 / 30000.0))
MASS = 0.01
GRAVITY = (0.0, float(np.float32(-9.81 * MASS)), 0.0)
DRAG, LIFT = float(np.float32(0.6)), float(np.float32(0.3))
RESTITUTION, FRICTION = float(np.float32(0.3)), float(np.float32(0.2))
WIND = (2.0, 0.0, 1.0)
K_TENSILE, K_SHEAR, K_BEND, DAMP = 500.0, 250.0, 50.0, 0.5
RATIO = 10  # fine steps per coarse step of the surrogate
LR = 1e-3
GROWTH, MAX_STRAIN = 0.05, 1000.0


def listed():
    return [
        # the reference's demo cloth in an interactive loop: one step, the points back to the host
        {"name": "interactive_20", "kind": "cloth", "rows": 20, "cols": 20, "rk4": True, "steps": 1,
         "read": "points", "woven": False},
        # one rendered frame of the small benchmark cloth: a frame's worth of steps, positions to the host
        {"name": "frame_32", "kind": "cloth", "rows": 32, "cols": 32, "rk4": False, "steps": 16,
         "read": "vertices", "woven": False},
        # a frame of a garment panel whose sides fill no tile, rendered from device memory
        {"name": "frame_157x211", "kind": "cloth", "rows": 157, "cols": 211, "rk4": True, "steps": 16,
         "read": "export", "woven": False},
        # a host solver that owns the state: write it, one step, read it back
        {"name": "exchange_500", "kind": "cloth", "rows": 500, "cols": 500, "rk4": False, "steps": 1,
         "read": "exchange", "woven": False},
        # the large benchmark cloth (plane and sphere), positions read back every few steps
        {"name": "cloth_1024", "kind": "cloth", "rows": 1024, "cols": 1024, "rk4": False, "steps": 16,
         "read": "pinned", "woven": True},
        # a sleeve: an arbitrary triangle mesh, so the general gather
        {"name": "tube_360x280", "kind": "tube", "rows": 360, "sectors": 280, "f64": False, "steps": 10},
        # the same step rerun in double precision, as it is used to state rounding error
        {"name": "tube_f64_90x61", "kind": "tube", "rows": 90, "sectors": 61, "f64": True, "steps": 10},
        # a few small cloths advanced a little at a time (control, reinforcement learning)
        {"name": "batch_24_small", "kind": "batch", "cloths": 24, "lo": 16, "hi": 48, "steps": 10},
        # dataset generation: a rollout of many uneven cloths
        {"name": "batch_256_rollout", "kind": "batch", "cloths": 256, "lo": 16, "hi": 128, "steps": 100},
        # checked surrogate rollout of uneven cloths from a given state, and the state back
        {"name": "coarse_48", "kind": "coarse", "cloths": 48, "lo": 16, "hi": 128, "coarse": 20},
        # the same on one large cloth
        {"name": "coarse_512", "kind": "coarse", "cloths": 1, "lo": 512, "hi": 512, "coarse": 20},
        # the surrogate's training loop at its default batch
        {"name": "train_65536", "kind": "train", "cloths": 8, "side": 160, "batch": 65536, "steps": 8},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["cloth", "cloth", "cloth", "tube", "batch", "batch", "coarse", "train"])
    if kind == "cloth":
        woven = rng.random() < 0.25
        return {"kind": "cloth", "rows": _log(rng, 8, 900), "cols": _log(rng, 8, 900), "rk4": rng.random() < 0.4,
                "steps": _log(rng, 1, 16),
                "read": rng.choice(["points", "vertices", "pinned", "exchange"] + ([] if woven else ["export"])),
                "woven": woven}
    if kind == "tube":
        f64 = rng.random() < 0.3
        return {"kind": "tube", "rows": _log(rng, 10, 90 if f64 else 360), "sectors": _log(rng, 8, 61 if f64 else 280),
                "f64": f64, "steps": _log(rng, 1, 10)}
    if kind == "batch":
        lo = _log(rng, 8, 40)
        return {"kind": "batch", "cloths": _log(rng, 2, 200), "lo": lo, "hi": lo + _log(rng, 1, 80),
                "steps": _log(rng, 1, 100)}
    if kind == "coarse":
        lo = _log(rng, 16, 96)
        return {"kind": "coarse", "cloths": _log(rng, 1, 32), "lo": lo, "hi": lo + _log(rng, 1, 32),
                "coarse": _log(rng, 2, 20)}
    return {"kind": "train", "cloths": rng.randint(1, 8), "side": _log(rng, 24, 160),
            "batch": 128 * _log(rng, 8, 512), "steps": _log(rng, 1, 8)}


# ---- scenes ------------------------------------------------------------------


def _rng(seed, salt):
    return np.random.default_rng([int(seed), int(salt)])


def _f32(x):
    return float(np.float32(x))


def _plane(y=-1.5, half=3.0):
    return (np.array([[-half, y, half], [half, y, half], [half, y, -half], [-half, y, -half]], np.float32),
            np.array([0, 1, 2, 0, 2, 3], np.uint32))


def _sphere(centre, radius=0.3, sectors=32, stacks=16):
    i, j = np.meshgrid(np.arange(stacks + 1), np.arange(sectors + 1), indexing="ij")
    lat, lon = math.pi / 2 - i * math.pi / stacks, j * 2 * math.pi / sectors
    pos = np.stack([np.cos(lat) * np.cos(lon), np.cos(lat) * np.sin(lon), np.sin(lat)], -1).reshape(-1, 3)
    idx = []
    for a in range(stacks):
        for b in range(sectors):
            p, q = a * (sectors + 1) + b, (a + 1) * (sectors + 1) + b
            idx += ([p, q, p + 1] if a else []) + ([p + 1, q, q + 1] if a + 1 < stacks else [])
    return (np.asarray(centre) + radius * pos).astype(np.float32), np.array(idx, np.uint32)


def _grid_rest(rows, cols, s):
    """Cloth::new's positions for spacing s at the origin, in f32."""
    s = np.float32(s)
    x = np.arange(cols, dtype=np.float32) * s - np.float32(cols) / np.float32(2) * s
    y = np.arange(rows, dtype=np.float32) * s - np.float32(rows) / np.float32(2) * s
    p = np.zeros((rows, cols, 3), np.float32)
    p[:, :, 0], p[:, :, 1] = x[None, :], y[:, None]
    return p.reshape(-1, 3)


def _grid_faces(rows, cols):
    i = (np.arange(rows - 1)[:, None] * cols + np.arange(cols - 1)[None, :]).ravel()
    a = np.stack([i + 1, i + cols, i], 1)
    b = np.stack([i + 1, i + cols + 1, i + cols], 1)
    return np.concatenate([a, b])


def _grid_struts(rows, cols):
    """Strut vertex pairs and class (0 tensile, 1 shear, 2 binding) of a Cloth::new grid."""
    v = np.arange(rows * cols).reshape(rows, cols)
    out = [(v[:, :-1], v[:, 1:], 0), (v[:-1], v[1:], 0), (v[:-1, 1:], v[1:, :-1], 1)]
    if rows > 2 and cols > 2:
        out += [(v[:-2, :-2], v[:-2, 2:], 2), (v[:-2, :-2], v[2:, :-2], 2)]
    return (np.concatenate([np.stack([a.ravel(), b.ravel()], 1) for a, b, _ in out]),
            np.concatenate([np.full(a.size, k) for a, _, k in out]))


def _billow(rest, seed, salt):
    """A state: the rest positions bulging out of plane, with a little noise and some velocity."""
    g = _rng(seed, salt)
    ext = np.maximum(rest.max(0) - rest.min(0), 1e-6)
    u = (rest - rest.min(0)) / ext
    amp, ph = g.uniform(0.02, 0.05) * ext.max(), g.uniform(0, math.pi)
    bulge = amp * np.sin(math.pi * u[:, 0] + ph) * np.sin(math.pi * u[:, 1])
    p = rest.astype(np.float64) + g.normal(0.0, 1e-5 * ext.max(), rest.shape)
    p[:, 2] += bulge
    v = g.normal(0.0, 0.02, rest.shape) + g.normal(0.0, 0.2, (1, 3)) * np.sin(math.pi * u[:, 1:2])
    pts = np.zeros((len(rest), 10), np.float32)
    pts[:, 0], pts[:, 1:4], pts[:, 4:7] = MASS, p, v
    return pts


def _wind(seed, salt):
    g = _rng(seed, salt)
    d = g.normal(size=3)
    return tuple(_f32(x) for x in d / np.linalg.norm(d) * g.uniform(0.0, 5.0))


def _jitter(ab, seed):
    """Per-strut stiffness factor in [0.9, 1.1), from the vertex pair."""
    h = ab[:, 0].astype(np.uint64) * np.uint64(0x9E3779B97F4A7C15) + ab[:, 1].astype(np.uint64)
    h = (h ^ np.uint64(int(seed) + 1)) * np.uint64(0xBF58476D1CE4E5B9)
    h = (h ^ (h >> np.uint64(31))) * np.uint64(0x94D049BB133111EB)
    return 0.9 + 0.2 * ((h >> np.uint64(40)).astype(np.float64) / 2.0 ** 24)


def _scene(rows, cols, seed, salt, factor=1.0, woven=False, wind=WIND, pins=None):
    """Plain description of one grid cloth, 1 m on its longer side."""
    s = _f32(1.0 / (max(rows, cols, 2) - 1))
    d = {"rows": rows, "cols": cols, "s": s, "wind": wind, "woven": woven, "seed": seed, "factor": factor,
         "rest": _grid_rest(rows, cols, s), "obstacles": [_plane()]}
    n = rows * cols
    d["pins"] = np.array([n - cols, n - 1] if pins is None else pins, np.uint32)
    if woven:
        d["pins"] = np.arange(n - cols, n, dtype=np.uint32)
        d["rest"] = (d["rest"].astype(np.float64) + _rng(seed, salt + 1).normal(0.0, s, (n, 3))).astype(np.float32)
        c = d["rest"].astype(np.float64).mean(0)
        d["obstacles"].append(_sphere((c[0], c[1] - 0.5, c[2])))
        d["points"] = np.zeros((n, 10), np.float32)
        d["points"][:, 0], d["points"][:, 1:4] = MASS, d["rest"]
        d["points"][:, 4:7] = _rng(seed, salt + 2).normal(0.0, 0.02, (n, 3))
    else:
        d["points"] = _billow(d["rest"], seed, salt)
    return d


def _nominal(d):
    """Cloth::new's constants: per-strut value times the nominal length of the class."""
    s, f = d["s"], d["factor"]
    lt, ls, lb = s, s * math.sqrt(2.0), 2.0 * s
    return [_f32(f * x) for x in (K_TENSILE * lt, DAMP * lt, K_SHEAR * ls, DAMP * ls, K_BEND * lb, DAMP * lb)]


def _woven_params(ab, cls, seed):
    k = np.array([K_TENSILE, K_SHEAR, K_BEND])[cls] * _jitter(ab, seed)
    return k.astype(np.float32), np.full(len(ab), DAMP, np.float32)


def _build_cloth(d):
    rows, cols = d["rows"], d["cols"]
    if not d["woven"]:
        mesh = fgb.Cloth.new(rows, cols, d["s"], (0.0, 0.0, 0.0), MASS, *_nominal(d), d["pins"]).mesh
    else:
        mesh = fgb.SpringyMesh.new(d["rest"], _grid_faces_ref(rows, cols), MASS * rows * cols, 1.0, 1.0,
                                   build_on_device=True)
        mesh.add_pins(d["pins"])
        v = np.arange(rows * cols).reshape(rows, cols)[:-2, :-2].ravel()
        mesh.add_struts(np.stack([np.stack([v, v + 2], 1), np.stack([v, v + 2 * cols], 1)], 1).reshape(-1, 2), 1.0, 1.0)
        _, ab = mesh.get_struts()
        ab = np.sort(ab.astype(np.int64), 1)
        step = ab[:, 1] - ab[:, 0]
        cls = np.where((step == 2) | (step == 2 * cols), 2, np.where((step == cols) | (step == 1), 0, 1))
        mesh.set_strut_params(*_woven_params(ab, cls, d["seed"]))
    mesh.set_points(d["points"])
    return mesh


def _grid_faces_ref(rows, cols):
    """The triangle list in the order Cloth::new makes it."""
    return _grid_faces(rows, cols).reshape(-1).astype(np.uint32)


def _config(rk4=False, wind=WIND):
    return fgb.Config.make(integration=1 if rk4 else 0, dt=DT, gravity=GRAVITY, wind=wind, lift_coefficient=LIFT,
                           drag_coefficient=DRAG, coefficient_of_restitution=RESTITUTION,
                           coefficient_of_friction=FRICTION)


def _tube(case, seed):
    """A sleeve of radius 0.15 m and length 0.5 m, both ends open, one end pinned."""
    R, S = case["rows"], case["sectors"]
    r, s = np.meshgrid(np.arange(R), np.arange(S), indexing="ij")
    a = 2 * math.pi * s / S
    pos = np.stack([0.15 * np.cos(a), 0.5 * r / max(R - 1, 1), 0.15 * np.sin(a)], -1).reshape(-1, 3).astype(np.float32)
    i = r[:-1] * S + s[:-1]
    j = r[:-1] * S + (s[:-1] + 1) % S
    f = np.concatenate([np.stack([i, i + S, j], -1).reshape(-1, 3), np.stack([j, i + S, j + S], -1).reshape(-1, 3)])
    g = _rng(seed, 3)
    pts = np.zeros((len(pos), 10), np.float32)
    pts[:, 0] = _f32(MASS * len(pos)) / np.float32(len(pos))
    pts[:, 1:4] = pos + g.normal(0.0, 1e-5, pos.shape)
    pts[:, 4:7] = g.normal(0.0, 0.02, pos.shape) + g.normal(0.0, 0.2, (1, 3))
    return {"rest": pos, "faces": f, "points": pts, "k": 2.0, "c": 0.005, "pins": np.arange(S, dtype=np.uint32),
            "wind": _wind(seed, 4), "obstacles": [_plane(-0.6), _sphere((0.0, 0.25, 0.0), 0.1, 16, 8)]}


def _batch(case, seed):
    out = []
    # sides come from the case alone, so that every seed has the same shapes
    sides = np.random.default_rng(case["cloths"] * 1000 + case["lo"]).integers(case["lo"], case["hi"] + 1, case["cloths"])
    for c, n in enumerate(sides):
        n, g = int(n), _rng(seed, 10 * c + 5)
        corners = [n * n - n, n * n - 1, 0, n - 1]
        kind = int(g.integers(0, 3))
        pins = ([corners[int(g.integers(0, 4))]] if kind == 0 else
                [int(x) for x in g.choice(corners, 2, replace=False)] if kind == 1 else list(range(n * n - n, n * n)))
        out.append(_scene(n, n, seed, 10 * c, factor=float(g.uniform(0.5, 2.0)), wind=_wind(seed, 10 * c + 6), pins=pins))
    return out


def _network(seed):
    """A surrogate in the shape training leaves it: weights, and the scales it standardises by."""
    g = _rng(seed, 77)
    h, f = 128, fgb.N_FEATURES
    w = [g.uniform(-1, 1, (h, f)) * math.sqrt(6 / (f + h)), g.normal(0, 0.1, h), g.uniform(-1, 1, (h, h)) * math.sqrt(3 / h),
         g.normal(0, 0.1, h), g.uniform(-1, 1, (3, h)) * math.sqrt(6 / (h + 3)), g.normal(0, 0.1, 3)]
    mean, std = np.zeros(f), np.ones(f)
    std[0:24], std[24:48], std[49:52], mean[52] = 0.02, 0.002, 0.05, 0.5
    return (np.concatenate([x.ravel() for x in w]).astype(np.float32), mean.astype(np.float32), std.astype(np.float32),
            np.array([0.0, -1e-4, 0.0], np.float32), np.full(3, 5e-5, np.float32))


_STREAM = None


def _stream():
    """The stream of the program around the simulation."""
    global _STREAM
    if _STREAM is None:
        _STREAM = torch.cuda.Stream()
    return _STREAM.cuda_stream


def _pinned(*shape):
    return torch.empty(shape, dtype=torch.float32, pin_memory=True).numpy()


def _collidables(obstacles):
    return [fgb.CollidableMesh.new(p, i) for p, i in obstacles]


def prepare(case, seed):
    st = {"case": case, "keep": []}
    kind = case["kind"]
    if kind == "cloth":
        d = _scene(case["rows"], case["cols"], seed, 0, woven=case["woven"], wind=_wind(seed, 9))
        st["meshes"] = [_build_cloth(d)]
        obstacles, cfg = d["obstacles"], _config(case["rk4"], d["wind"])
        n = case["rows"] * case["cols"]
        if case["read"] == "pinned":
            st["out"] = _pinned(n, 3)
        elif case["read"] == "exchange":
            st["in"], st["out"] = _pinned(n, 10), _pinned(n, 10)
            st["in"][:] = d["points"]
        elif case["read"] == "export":
            st["out"] = torch.empty((n, 9), dtype=torch.float32, device="cuda")
    elif kind == "tube":
        d = _tube(case, seed)
        m = fgb.SpringyMesh.new(d["rest"], d["faces"].astype(np.uint32), _f32(MASS * len(d["rest"])), d["k"], d["c"])
        m.add_pins(d["pins"])
        m.set_points(d["points"])
        if case["f64"]:
            m.set_precision(64)
        st["meshes"] = [m]
        obstacles, cfg = d["obstacles"], _config(False, d["wind"])
    else:
        if kind == "train":
            scenes = [_scene(case["side"], case["side"], seed, 10 * c, wind=_wind(seed, 10 * c + 6))
                      for c in range(case["cloths"])]
        else:
            scenes = _batch(case, seed)
        st["meshes"] = []
        for d in scenes:
            m = _build_cloth(d)
            m.set_wind(d["wind"])
            st["meshes"].append(m)
        obstacles, cfg = [_plane()], _config()
        ends = np.cumsum([d["rows"] * d["cols"] for d in scenes])
        st["at"] = list(zip([0] + [int(e) for e in ends[:-1]], [int(e) for e in ends]))
        total = int(ends[-1])
        if kind == "batch":
            st["out"] = torch.empty((total, 9), dtype=torch.float32, device="cuda")
        elif kind == "coarse":
            st["in"], st["out"] = _pinned(total, 10), _pinned(total, 10)
            st["in"][:] = np.concatenate([d["points"] for d in scenes])
    st["obstacles"] = _collidables(obstacles)
    sim = st["sim"] = fgb.Simulation.new(st["meshes"], st["obstacles"])
    sim.set_config(cfg)
    sim.set_stream(_stream())
    sim.step(0)  # set-up: the state, the topology and the obstacles go to the device
    if kind == "coarse":
        net = _network(seed)
        st["net"] = fgb.Surrogate.new(seed)
        st["net"].set_params(net[0])
        st["net"].set_normalization(*net[1:])
        st["check"] = fgb.SurrogateCheck.make(energy_growth=GROWTH, max_strain=MAX_STRAIN)
    elif kind == "train":
        net = st["net"] = fgb.Surrogate.new(seed)
        net.set_params(_network(seed)[0])
        net.reserve(total)
        net.collect(sim, RATIO, 1)
        net.fit_normalization()
        st["epoch"] = 0
    return st


def run(state):
    case, sim, kind = state["case"], state["sim"], state["case"]["kind"]
    if kind == "cloth":
        mesh = state["meshes"][0]
        if case["read"] == "exchange":
            mesh.set_points(state["in"])
        sim.step(case["steps"])
        if case["read"] in ("points", "exchange"):
            return mesh.get_points(state.get("out"))
        if case["read"] in ("vertices", "pinned"):
            return mesh.get_positions(state.get("out"))
        mesh.export_vertices(state["out"].data_ptr(), stream_handle=_stream())
        return state["out"]
    if kind == "tube":
        mesh = state["meshes"][0]
        sim.step(case["steps"])
        return mesh.get_points_f64() if case["f64"] else mesh.get_points()
    if kind == "batch":
        sim.step(case["steps"])
        for m, (a, _) in zip(state["meshes"], state["at"]):
            m.export_vertices(state["out"].data_ptr() + 36 * a, stream_handle=_stream())
        return state["out"]
    if kind == "coarse":
        for m, (a, b) in zip(state["meshes"], state["at"]):
            m.set_points(state["in"][a:b])
        back = sim.step_surrogate(state["net"], RATIO, case["coarse"], state["check"])
        for m, (a, b) in zip(state["meshes"], state["at"]):
            m.get_points(state["out"][a:b])
        return {"points": state["out"], "fallbacks": back}
    losses = state["net"].train(case["steps"], case["batch"], LR, state["epoch"])
    state["epoch"] += 1
    return {"losses": losses, "params": state["net"].get_params()}


def _counts(case):
    """Vertices, struts and faces of a case's meshes."""
    if case["kind"] == "tube":
        r, s = case["rows"], case["sectors"]
        return r * s, r * s + 2 * (r - 1) * s, 2 * (r - 1) * s
    if case["kind"] == "cloth":
        grids = [(case["rows"], case["cols"])]
    elif case["kind"] == "train":
        grids = [(case["side"],) * 2] * case["cloths"]
    else:
        g = np.random.default_rng(case["cloths"] * 1000 + case["lo"]).integers(case["lo"], case["hi"] + 1, case["cloths"])
        grids = [(int(n), int(n)) for n in g]
    v = sum(r * c for r, c in grids)
    s = sum(r * (c - 1) + (r - 1) * c + (r - 1) * (c - 1) + 2 * max(r - 2, 0) * max(c - 2, 0) for r, c in grids)
    return v, s, sum(2 * (r - 1) * (c - 1) for r, c in grids)


def work(case):
    """Bytes: the state and the strut constants once in, the result once out.  Operations: one step takes
    about 36 per strut, 120 per face and 40 per vertex; the network 47,360 per vertex forward."""
    v, s, f = _counts(case)
    step = 36 * s + 120 * f + 40 * v
    if case["kind"] == "train":
        rows = case["batch"] * case["steps"]
        return {"bytes": rows * (54 + 3) * 4 + 2 * fgb.N_PARAMS * 4, "flops": rows * 3 * 47360}
    if case["kind"] == "coarse":
        return {"bytes": v * (40 + 40 + 16) + 12 * s, "flops": case["coarse"] * v * (47360 + 300)}
    state = 28 * (2 if case.get("f64") else 1)
    out = {"points": 40, "exchange": 40, "vertices": 12, "pinned": 12, "export": 36}.get(
        case.get("read"), 36 if case["kind"] == "batch" else 80 if case.get("f64") else 40)
    return {"bytes": v * (state + out) + 12 * s, "flops": case["steps"] * step}


# ---- the same in 64 bits, in plain torch ----------------------------------------

_DEV = "cuda" if torch.cuda.is_available() else "cpu"


def _t(x):
    return torch.as_tensor(np.asarray(x, np.float64), device=_DEV)


def _i(x):
    return torch.as_tensor(np.asarray(x, np.int64), device=_DEV)


def _norm(x):
    return x.square().sum(-1).sqrt()


class _Exact:
    """One mesh in 64 bits: struts, faces, integration and collisions as the reference defines them."""

    def __init__(self, rest, ab, kc, faces, pins, points, wind, obstacles, rk4=False):
        self.a, self.b, self.faces = _i(ab[:, 0]), _i(ab[:, 1]), _i(faces)
        rest = _t(rest)
        self.rest = rest
        self.L = _norm(rest[self.a] - rest[self.b])
        k, c, scaled = kc
        self.k, self.c = (_t(k) / self.L, _t(c) / self.L) if scaled else (_t(k), _t(c))
        self.free = torch.ones(len(rest), dtype=torch.bool, device=_DEV)
        self.free[_i(pins)] = False
        pts = _t(points)
        self.m, self.p, self.v = pts[:, 0:1], pts[:, 1:4].clone(), pts[:, 4:7].clone()
        self.wind, self.g, self.rk4 = _t(wind), _t(GRAVITY), rk4
        fv = [_t(p)[_i(i).reshape(-1, 3)] for p, i in obstacles]
        o = self.obs = torch.cat(fv)
        n = torch.linalg.cross(o[:, 1] - o[:, 0], o[:, 2] - o[:, 0])
        n = self.on = n / _norm(n)[:, None]
        x, y, z = n.unbind(-1)
        self.axis = torch.where((x >= y) & (x >= z), 0, torch.where((y >= x) & (y >= z), 1, 2))

    def forces(self):
        p, v = self.p, self.v
        F = self.g.expand_as(p).clone()
        d = p[self.b] - p[self.a]
        ln = _norm(d)
        u = d / ln[:, None]
        f = (self.k * (ln - self.L) + self.c * ((v[self.b] - v[self.a]) * u).sum(-1))[:, None] * u
        F.index_add_(0, self.a, f)
        F.index_add_(0, self.b, -f)
        x, w = p[self.faces], v[self.faces]
        rv = w.mean(1) - self.wind
        cr = torch.linalg.cross(x[:, 1] - x[:, 0], x[:, 2] - x[:, 0])
        ln = _norm(cr)
        n = cr / ln[:, None]
        eff = ln / 2 * (n * rv).sum(-1).abs()
        tot = -(eff * (DRAG + LIFT * _norm(torch.linalg.cross(n, rv))))[:, None] * rv
        for k in range(3):
            e, g = x[:, (k + 2) % 3] - x[:, k], x[:, (k + 1) % 3] - x[:, k]
            share = torch.atan2(_norm(torch.linalg.cross(e, g)), (e * g).sum(-1)) / math.pi
            F.index_add_(0, self.faces[:, k], share[:, None] * tot)
        return F

    def step(self):
        F = self.forces()
        acc, p, v, h = F / self.m, self.p, self.v, DT
        if self.rk4:
            np_ = p + h / 6 * v + h / 3 * (v + acc * (h / 2)) * 2 + h / 6 * (v + acc * h)
        else:
            np_ = p + v * h
        self.settle(np_, v + acc * h, F, h)

    def settle(self, np_, nv, F, h):
        """update_points: the first face crossed, its response, pins restored."""
        p, v = self.p, self.v
        best = torch.full((len(p),), len(self.obs), dtype=torch.long, device=_DEV)
        for f0 in range(0, len(self.obs), 32):
            n, o = self.on[f0:f0 + 32], self.obs[f0:f0 + 32]
            off = (o[:, 0] * n).sum(-1)
            d0, d1 = p @ n.T - off, np_ @ n.T - off
            vi, fi = torch.nonzero(torch.signbit(d0) != torch.signbit(d1), as_tuple=True)
            if not len(vi):
                continue
            e0, e1 = d0[vi, fi], d1[vi, fi]
            cp = p[vi] + (e0 / (e0 - e1))[:, None] * (np_[vi] - p[vi])
            keep = torch.ones((len(vi), 3), dtype=torch.float64, device=_DEV)
            keep[torch.arange(len(vi), device=_DEV), self.axis[f0 + fi]] = 0.0
            tri, q, nn = o[fi] * keep[:, None, :], cp * keep, n[fi]
            side = [torch.signbit((torch.linalg.cross(tri[:, (k + 1) % 3] - tri[:, k], q - tri[:, k]) * nn).sum(-1))
                    for k in range(3)]
            hit = (side[0] == side[1]) & (side[1] == side[2])
            best.scatter_reduce_(0, vi[hit], f0 + fi[hit], "amin")
        hit = torch.nonzero(best < len(self.obs)).reshape(-1)
        if len(hit):
            n, o0 = self.on[best[hit]], self.obs[best[hit], 0]
            d0, d1 = ((p[hit] - o0) * n).sum(-1), ((np_[hit] - o0) * n).sum(-1)
            t = (h * d0 / (d0 - d1))[:, None]
            vc = v[hit] + t * F[hit] / self.m[hit]
            vn = (vc * n).sum(-1, keepdim=True) * n
            vt = vc - vn
            lt, ln = _norm(vt)[:, None], _norm(vn)[:, None]
            slide = torch.where(lt > 0, vt - vt / lt.clamp_min(1e-300) * torch.minimum(FRICTION * ln, lt), torch.zeros_like(vt))
            np_, nv = np_.clone(), nv.clone()
            np_[hit], nv[hit] = p[hit] + t * v[hit] + n * 1e-4, slide - vn * RESTITUTION
        self.p = torch.where(self.free[:, None], np_, p)
        self.v = torch.where(self.free[:, None], nv, v)

    def points(self):
        return torch.cat([self.m, self.p, self.v, torch.zeros_like(self.p)], 1)

    def vertices(self):
        """Render vertices: position, white, and the sum of the faces' normals, normalised."""
        x = self.p[self.faces]
        n = torch.linalg.cross(x[:, 0] - x[:, 1], x[:, 0] - x[:, 2])
        s = torch.zeros_like(self.p)
        for k in range(3):
            s.index_add_(0, self.faces[:, k], n)
        return torch.cat([self.p, torch.ones_like(self.p), s / _norm(s)[:, None]], 1)

    def features(self, rows, cols, T):
        """Surrogate inputs of a grid, unstandardised; and the scale s = T / h."""
        P, V, R0 = (a.reshape(rows, cols, 3) for a in (self.p, self.v, self.rest))
        h = _norm(R0[:, 1:] - R0[:, :-1]).mean()
        s = T / h
        pos, vel, near = [], [], {}
        for dr, dc in ((-1, -1), (-1, 0), (-1, 1), (0, -1), (0, 1), (1, -1), (1, 0), (1, 1)):
            r, c = torch.arange(rows, device=_DEV)[:, None] + dr, torch.arange(cols, device=_DEV)[None, :] + dc
            ok = ((r >= 0) & (r < rows) & (c >= 0) & (c < cols))[..., None]
            j = (r.clamp(0, rows - 1), c.clamp(0, cols - 1))
            pos.append(torch.where(ok, ((P[j] - P) - (R0[j] - R0)) / h, torch.zeros_like(P)))
            vel.append(torch.where(ok, (V[j] - V) * s, torch.zeros_like(P)))
            near[dr, dc] = torch.where(ok, P[j], P)
        n = torch.linalg.cross(near[0, 1] - near[0, -1], near[1, 0] - near[-1, 0])
        n = n / _norm(n)[..., None]
        pin = (~self.free).reshape(rows, cols, 1).double()
        ang = torch.stack([torch.acos(n[..., 1].clamp(-1, 1)), torch.atan2(n[..., 2], n[..., 0])], -1) / math.pi
        return torch.cat(pos + vel + [pin, (self.wind - V) * s, ang], -1).reshape(rows * cols, -1), s


def _gelu(x):
    return 0.5 * x * (1 + torch.tanh(math.sqrt(2 / math.pi) * (x + 0.044715 * x ** 3)))


def _unpack(flat):
    out, at = [], 0
    for shape in ((128, fgb.N_FEATURES), (128,), (128, 128), (128,), (3, 128), (3,)):
        n = int(np.prod(shape))
        out.append(_t(flat[at:at + n]).reshape(shape))
        at += n
    return out


def _forward(w, x):
    return _gelu(_gelu(x @ w[0].T + w[1]) @ w[2].T + w[3]) @ w[4].T + w[5]


def _grid_parts(d):
    ab, cls = _grid_struts(d["rows"], d["cols"])
    if d["woven"]:
        return ab, _woven_params(np.sort(ab, 1), cls, d["seed"]) + (False,)
    nom = np.array(_nominal(d)).reshape(3, 2)
    return ab, (nom[cls, 0], nom[cls, 1], True)


def _exact_grid(d, rk4=False):
    ab, kc = _grid_parts(d)
    return _Exact(d["rest"], ab, kc, _grid_faces(d["rows"], d["cols"]), d["pins"], d["points"], d["wind"],
                  d["obstacles"], rk4)


def _exact_batch(scenes):
    """All cloths of a batch as one mesh of separate parts, each face with its cloth's wind."""
    at, parts = 0, []
    for d in scenes:
        ab, kc = _grid_parts(d)
        f = _grid_faces(d["rows"], d["cols"])
        parts.append((d["rest"], ab + at, kc[0], kc[1], f + at, d["pins"].astype(np.int64) + at, d["points"],
                      np.broadcast_to(d["wind"], (len(f), 3))))
        at += len(d["rest"])
    rest, ab, k, c, f, pins, pts, wind = (np.concatenate(x) for x in zip(*parts))
    return _Exact(rest, ab, (k, c, True), f, pins, pts, wind, scenes[0]["obstacles"])


def exact(case, seed):
    kind = case["kind"]
    if kind == "cloth":
        d = _scene(case["rows"], case["cols"], seed, 0, woven=case["woven"], wind=_wind(seed, 9))
        e = _exact_grid(d, case["rk4"])
        for _ in range(case["steps"]):
            e.step()
        return {"points": e.points, "exchange": e.points, "export": e.vertices}.get(case["read"], lambda: e.p)()
    if kind == "tube":
        d = _tube(case, seed)
        ab = np.unique(np.sort(np.concatenate([d["faces"][:, [0, 1]], d["faces"][:, [1, 2]], d["faces"][:, [2, 0]]]), 1), axis=0)
        kc = (np.full(len(ab), _f32(d["k"])), np.full(len(ab), _f32(d["c"])), True)
        e = _Exact(d["rest"], ab, kc, d["faces"], d["pins"], d["points"], d["wind"], d["obstacles"])
        for _ in range(case["steps"]):
            e.step()
        return e.points()
    if kind == "batch":
        e = _exact_batch(_batch(case, seed))
        for _ in range(case["steps"]):
            e.step()
        return e.vertices()
    T = RATIO * DT
    if kind == "coarse":
        flat, mean, std, om, os_ = _network(seed)
        w, out = _unpack(flat), []
        for d in _batch(case, seed):
            e = _exact_grid(d)
            for _ in range(case["coarse"]):
                f, s = e.features(d["rows"], d["cols"], T)
                dv = (_forward(w, (f - _t(mean)) / _t(std)) * _t(os_) + _t(om)) / s
                nv = e.v + dv
                e.settle(e.p + (e.v + nv) * (0.5 * T), nv, dv * e.m / T, T)
            out.append(e.points())
        return {"points": torch.cat(out), "fallbacks": None}
    feats, tgts = [], []
    for c in range(case["cloths"]):
        d = _scene(case["side"], case["side"], seed, 10 * c, wind=_wind(seed, 10 * c + 6))
        e = _exact_grid(d)
        f, s = e.features(d["rows"], d["cols"], T)
        v0 = e.v
        for _ in range(RATIO):
            e.step()
        feats.append(f)
        tgts.append((e.v - v0) * s)
    X, Y = torch.cat(feats), torch.cat(tgts)

    def scales(x):
        sd = (x.square().mean(0) - x.mean(0).square()).clamp_min(0).sqrt()
        return x.mean(0), torch.where(sd < 1e-6, torch.ones_like(sd), sd)

    (xm, xs), (ym, ys) = scales(X), scales(Y)
    w = [x.requires_grad_() for x in _unpack(_network(seed)[0])]
    m, v = [torch.zeros_like(x) for x in w], [torch.zeros_like(x) for x in w]
    losses, mask = [], (1 << 64) - 1
    for k in range(case["steps"]):
        base = np.uint64((k * 0x9E3779B97F4A7C15) & mask)  # the first pass draws with seed 0
        z = (np.arange(case["batch"], dtype=np.uint64) * np.uint64(0x9E3779B97F4A7C15)) ^ base
        for shift, mul in ((30, 0xBF58476D1CE4E5B9), (27, 0x94D049BB133111EB)):
            z = (z ^ (z >> np.uint64(shift))) * np.uint64(mul)
        row = _i(((z ^ (z >> np.uint64(31))) % np.uint64(len(X))).astype(np.int64))
        loss = (_forward(w, (X[row] - xm) / xs) - (Y[row] - ym) / ys).square().mean()
        grad = torch.autograd.grad(loss, w)
        losses.append(loss.detach())
        with torch.no_grad():
            for x, g, a, b in zip(w, grad, m, v):
                a.mul_(0.9).add_(g, alpha=0.1)
                b.mul_(0.999).addcmul_(g, g, value=0.001)
                x -= LR * (a / (1 - 0.9 ** (k + 1))) / ((b / (1 - 0.999 ** (k + 1))).sqrt() + 1e-8)
    return {"losses": torch.stack(losses), "params": torch.cat([x.detach().reshape(-1) for x in w])}
