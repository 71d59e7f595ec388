"""The measured workloads of the DEM framework: what its users have it do, through its public calls.

Every case is a specimen that a script set up (particles, groups, walls) and a pass over it: some
timesteps and the read-back of the state into the caller's pinned host arrays, as a driver's loop
does.  A pass goes on from the state the one before left, so neighbour searches, wear of the bonds
and wall motion fall where they fall in a run.  The kinds:

  gravity   non-rotational elastic spheres in a six-walled box under gravity with damping
  pack      dense rotational frictional packing between two walls, damped
  shear     loose frictional shear cell, periodic in x, moving walls, a load servo on the top one
  flow      dense frictional packing with a neighbour search every few steps (fast flow)
  slide     loose non-rotational cell under the NRotFriction law
  block     bonded rock block under platens, failures handed to the friction group on the device
  ensemble  many bonded cylinders of different sizes advanced together
  window    differentiable loading window: forward, reverse pass and rewind

``exact`` restates the physics in plain torch at 64 bits (contact forces need only the touching
pairs, so it uses one generous pair list per pass and no neighbour-search bookkeeping but the
periodic wrap).
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.getcwd(), "esys-particle_b200"))
from esys.lsm import _capi  # noqa: E402
from esys.lsm import geometry  # noqa: E402

PI_REF = 3.141592654  # the pi of the particles' masses and the walls' stiffness


def listed():
    return [
        # the smallest call: a test-sized frictional packing stepped between a script's own actions
        {"name": "pack_180_f64", "kind": "pack", "nx": 6, "ny": 5, "nz": 6, "precision": 64, "steps": 20},
        # a tutorial-sized packing, odd sides, in the FP32-force form
        {"name": "pack_6k_f32", "kind": "pack", "nx": 19, "ny": 17, "nz": 21, "precision": 32, "steps": 50},
        # the 8,000-sphere gravity packing configuration
        {"name": "gravity_8k_f64", "kind": "gravity", "side": 20, "layers": 20, "precision": 64, "steps": 100},
        # a production shear cell (the 250,000-sphere configuration) in both precision forms
        {"name": "shear_250k_f32", "kind": "shear", "count": 31250, "block": 12.5, "tx": 2, "ty": 2, "tz": 2,
         "precision": 32, "steps": 200},
        {"name": "shear_250k_f64", "kind": "shear", "count": 31250, "block": 12.5, "tx": 2, "ty": 2, "tz": 2,
         "precision": 64, "steps": 200},
        # a shear cell of the size a parameter study repeats, odd count
        {"name": "shear_31k_f32", "kind": "shear", "count": 30977, "block": 12.5, "tx": 1, "ty": 1, "tz": 1,
         "precision": 32, "steps": 100},
        # fast dense flow: the neighbour search is as much of the work as the steps
        {"name": "flow_100k_f64", "kind": "flow", "nx": 48, "ny": 41, "nz": 51, "precision": 64, "every": 10,
         "searches": 4},
        # non-rotational spheres under the widened friction law
        {"name": "slide_62k_f64", "kind": "slide", "count": 31250, "block": 12.5, "tx": 2, "ty": 1, "tz": 1,
         "precision": 64, "steps": 100},
        # bonded rock: a laboratory-sized block in FP64, a large one in the FP32-force form
        {"name": "block_29k_f64", "kind": "block", "count": 29000, "tx": 1, "ty": 1, "tz": 1, "precision": 64,
         "steps": 50},
        {"name": "block_240k_f32", "kind": "block", "count": 30000, "tx": 2, "ty": 2, "tz": 2, "precision": 32,
         "steps": 20},
        # a batch of bonded cylinders (parameter sweep), FP32 forces, one launch per step for all
        {"name": "ensemble_12_f32", "kind": "ensemble", "specimens": 12, "low": 2000, "high": 24000,
         "precision": 32, "steps": 40},
        # gradients of platen reactions with respect to stiffnesses, damping and initial velocities
        {"name": "window_12k_f64", "kind": "window", "count": 12000, "precision": 64, "steps": 40, "every": 10},
    ]


def draw(rng):
    def log_int(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["gravity", "pack", "pack", "shear", "shear", "flow", "slide", "block", "block", "ensemble",
                       "window"])
    precision = rng.choice([32, 64])
    if kind == "gravity":
        s = log_int(6, 34)
        return {"kind": kind, "side": s, "layers": max(4, s + rng.randint(-3, 3)), "precision": precision,
                "steps": rng.randint(20, 120)}
    if kind == "pack":
        s = log_int(5, 40)
        return {"kind": kind, "nx": s + rng.randint(0, 3), "ny": s, "nz": max(4, s + rng.randint(-1, 2)),
                "precision": precision, "steps": rng.randint(10, 60)}
    if kind == "flow":
        s = log_int(12, 44)
        return {"kind": kind, "nx": s + rng.randint(0, 5), "ny": s, "nz": s + rng.randint(-3, 3),
                "precision": precision, "every": rng.randint(5, 20), "searches": rng.randint(1, 4)}
    if kind in ("shear", "slide"):
        c = log_int(2500, 31250)
        return {"kind": kind, "count": c, "block": 12.5 * (c / 31250.0) ** (1.0 / 3.0), "tx": rng.randint(1, 2),
                "ty": rng.randint(1, 2), "tz": rng.randint(1, 2), "precision": precision if kind == "shear" else 64,
                "steps": rng.randint(40, 200)}
    if kind == "block":
        return {"kind": kind, "count": log_int(1500, 30000), "tx": rng.randint(1, 2), "ty": rng.randint(1, 2),
                "tz": rng.randint(1, 2), "precision": precision, "steps": rng.randint(10, 50)}
    if kind == "ensemble":
        return {"kind": kind, "specimens": rng.randint(3, 16), "low": 2000, "high": log_int(3000, 24000),
                "precision": precision, "steps": rng.randint(10, 50)}
    return {"kind": kind, "count": log_int(1500, 12000), "precision": precision, "steps": rng.randint(10, 40),
            "every": rng.randint(5, 20)}


# ---------------------------------------------------------------------------
# specimens: plain arrays and parameters, shared by prepare() and exact()
# ---------------------------------------------------------------------------
def sphere_mass(rad):
    return (4.0 / 3.0) * PI_REF * rad ** 3


def lattice(nx, ny, nz):
    g = np.stack(np.meshgrid(np.arange(nx), np.arange(ny), np.arange(nz), indexing="ij"), -1)
    return g.reshape(-1, 3).astype(np.float64)


def tiled(pos, size, tx, ty, tz, mirror):
    """Copies of a packed block side by side; mirrored copies meet face to face."""
    out = []
    for t in ((a, b, c) for a in range(tx) for b in range(ty) for c in range(tz)):
        p = pos.copy()
        for k in range(3):
            p[:, k] = size[k] * (t[k] + 1) - p[:, k] if mirror and t[k] % 2 else size[k] * t[k] + p[:, k]
        out.append(p)
    return np.concatenate(out)


def gravity_specimen(c, rng):
    g = lattice(c["side"], c["side"], c["layers"])
    L, H = float(c["side"]), 2.0 * c["layers"]
    # settled enough to touch: layers 0.9 apart, as after the first fall
    pos = (g + 0.5) * np.array([1.0, 1.0, 0.9]) + rng.uniform(-0.05, 0.05, size=g.shape)
    rad = rng.uniform(0.4, 0.5, size=len(g))
    walls = [("xhi", (L, 0, 0), (-1, 0, 0)), ("xlo", (0, 0, 0), (1, 0, 0)), ("yhi", (0, L, 0), (0, -1, 0)),
             ("ylo", (0, 0, 0), (0, 1, 0)), ("zhi", (0, 0, H), (0, 0, -1)), ("zlo", (0, 0, 0), (0, 0, 1))]
    return dict(rot=False, grid=1.2, skin=0.2, lo=(0, 0, 0), hi=(L, L, H), periodic=False, dt=1e-4, pos=pos, rad=rad,
                vel=rng.normal(0.0, 0.1, size=pos.shape), law="elastic", k=1000.0, walls=walls, wall_k=1000.0,
                gravity=(0, 0, -9.81), damping=[(0, 0.01, 100)])


def pack_specimen(c, rng):
    g = lattice(c["nx"], c["ny"], c["nz"])
    a = 0.93
    pos = (g + 0.5) * a + rng.uniform(-0.03, 0.03, size=g.shape)
    rad = np.clip(np.exp(np.log(0.5) + 0.25 * rng.standard_normal(len(g))) * 0.5 + 0.25, 0.3, 0.5)
    hi = (c["nx"] * a, c["ny"] * a + 0.1, c["nz"] * a)
    v = 0.5
    return dict(rot=True, grid=1.2, skin=0.2, lo=(0, -0.1, 0), hi=hi, periodic=c["kind"] == "flow", dt=5e-5, pos=pos,
                rad=rad, vel=rng.normal(0, v, size=pos.shape), angvel=rng.normal(0, v, size=pos.shape), law="friction",
                k=1e4, ks=1e4, mu=0.6, walls=[("floor", (0, -0.1, 0), (0, 1, 0)), ("roof", (0, hi[1], 0), (0, -1, 0))],
                wall_k=1e4, damping=[(0, 0.002, 50), (1, 0.002, 50)])


def shear_specimen(c, rng):
    b = c["block"]
    size = (4.0 * b, 2.0 * b, 4.0 * b)
    pos, rad = geometry.rsi_pack(c["count"], (0, 0, 0), size, seed=int(rng.integers(1 << 30)), periodic_x=True,
                                 lognormal=(0.5, 0.25), rmin=0.2, rmax=1.0, max_attempts=5000)
    n = c["tx"] * c["ty"] * c["tz"]
    pos, rad = tiled(pos, size, c["tx"], c["ty"], c["tz"], False), np.tile(rad, n)
    order = np.argsort(-rad, kind="stable")  # the insertion order of one packing: largest first
    pos, rad = pos[order], rad[order]
    hi = (size[0] * c["tx"], size[1] * c["ty"], size[2] * c["tz"])
    shear = c["kind"] == "shear"
    return dict(rot=shear, grid=2.2, skin=0.2, lo=(0, 0, 0), hi=hi, periodic=True, dt=5e-5, pos=pos, rad=rad,
                vel=rng.normal(0, 0.1, size=pos.shape), angvel=rng.normal(0, 0.1, size=pos.shape) if shear else None,
                law="friction" if shear else "nfriction", k=1e4, ks=1e4, mu=0.6,
                walls=[("bottom", (0, 0, 0), (0, 1, 0)), ("top", (0, hi[1], 0), (0, -1, 0))], wall_k=1e4,
                wall_vel={"top": (0.01, 0, 0)}, servo=(0.0, -1e3, 0.0) if shear else None)


def fitted(count, seed):
    """A dense fitted packing in a b x 2b x b box and its touching pairs."""
    b = 66.0 * (count / 1e6) ** (1.0 / 3.0)
    pos, rad = geometry.fit_pack(count, (0, 0, 0), (b, 2 * b, b), 0.2, 1.0, seed=seed, max_failures=300)
    i, j = geometry.distance_connections(pos, rad, 1e-3)
    return pos, rad, i, j, (b, 2 * b, b)


def bond_arrays(i, j, order):
    """The pairs after the particles were put in `order`."""
    place = np.empty_like(order)
    place[order] = np.arange(len(order))
    return place[i], place[j]


def block_specimen(c, rng):
    pos, rad, i, j, size = fitted(c["count"], int(rng.integers(1 << 30)))
    m = len(rad)
    t = (c["tx"], c["ty"], c["tz"])
    nt = t[0] * t[1] * t[2]
    faces = []  # spheres that touch a shared face touch their own mirror image
    for k in range(3):
        step = (t[1] * t[2], t[2], 1)[k]
        for tile in range(nt):
            q = (tile // (t[1] * t[2]), tile // t[2] % t[1], tile % t[2])[k]
            if q + 1 < t[k]:
                gap = (size[k] - pos[:, k] if q % 2 == 0 else pos[:, k]) - rad
                s = np.nonzero(2 * gap <= 1e-3)[0]
                faces.append((s + m * tile, s + m * (tile + step)))
    off = np.arange(nt)[:, None] * m
    i = np.concatenate([(i + off).ravel()] + [f[0] for f in faces])
    j = np.concatenate([(j + off).ravel()] + [f[1] for f in faces])
    pos, rad = tiled(pos, size, *t, True), np.tile(rad, nt)
    order = rng.permutation(len(rad))  # a packer's insertion order is scattered in space
    i, j = bond_arrays(i, j, order)
    pos, rad = pos[order], rad[order]
    hi = tuple(size[k] * t[k] for k in range(3))
    return bonded(pos, rad, i, j, (0, 0, 0), hi, rng, dt=1e-5, kn=1e5, ks=1e5, strength=(0.5, 1.0, 1.0, 0.5),
                  rate=1e-9, damping=[], friction=True)


def bonded(pos, rad, i, j, lo, hi, rng, *, dt, kn, ks, strength, rate, damping, friction, vel=1e-3, speed=None):
    y0, y1 = float((pos[:, 1] - rad).min()), float((pos[:, 1] + rad).max())
    v = 0.5 * rate * (y1 - y0) / dt if speed is None else speed  # each platen, `rate` of the height per step
    return dict(rot=True, grid=2.2, skin=0.2, lo=lo, hi=hi, periodic=False, dt=dt, pos=pos, rad=rad,
                vel=rng.normal(0, vel, size=pos.shape), angvel=rng.normal(0, vel, size=pos.shape),
                law="friction" if friction else None, k=kn, ks=ks, mu=0.6, bonds=(i, j), bond_k=(kn, ks, 1e3, 1e3),
                strength=strength, walls=[("bottom", (0, y0, 0), (0, 1, 0)), ("top", (0, y1, 0), (0, -1, 0))],
                wall_k=1e5, wall_vel={"bottom": (0, v, 0), "top": (0, -v, 0)}, damping=damping)


def ensemble_specimens(c, rng):
    """Cylinders (height four radii) of log-uniform sizes cut from one fitted block, the packing a program has on
    file; their stiffnesses, strengths and velocities are drawn."""
    out = []
    big = c["high"]
    R = (big / (2.2 * 4.0 * math.pi)) ** (1.0 / 3.0)
    pos, rad = geometry.fit_pack(int(2 * big) + 100, (-R, 0, -R), (R, 4 * R, R), 0.2, 1.0, seed=5, max_failures=300)
    sizes = np.random.default_rng(5)
    for _ in range(c["specimens"]):
        n = math.exp(sizes.uniform(math.log(c["low"]), math.log(big)))
        r = R * (n / big) ** (1.0 / 3.0)
        keep = (pos[:, 0] ** 2 + pos[:, 2] ** 2 <= r * r) & (pos[:, 1] <= 4 * r)
        p, a = pos[keep], rad[keep]
        i, j = geometry.distance_connections(p, a, 1e-3)
        kn, ks = np.exp(rng.uniform(math.log(1e4), math.log(1e5), size=2))
        sn, ss = np.exp(rng.uniform(math.log(0.5), math.log(2.0), size=2))
        out.append(bonded(p, a, i, j, (-r - 1, -1, -r - 1), (r + 1, 4 * r + 1, r + 1), rng, dt=1e-5, kn=kn, ks=ks,
                          strength=(sn, ss, ss, sn), rate=1e-7, damping=[(0, 0.01, 100), (1, 0.01, 100)],
                          friction=True))
    return out


def window_specimen(c, rng):
    pos, rad, i, j, size = fitted(c["count"], int(rng.integers(1 << 30)))
    return bonded(pos, rad, i, j, (0, 0, 0), size, rng, dt=1e-5, kn=1e5, ks=1e5, strength=(1e6,) * 4, rate=0.0,
                  speed=1.0, damping=[(0, 0.05, 100), (1, 0.05, 100)], friction=False, vel=0.01)


SPECIMEN = {"gravity": gravity_specimen, "pack": pack_specimen, "flow": pack_specimen, "shear": shear_specimen,
            "slide": shear_specimen, "block": block_specimen, "window": window_specimen}


def specimens(case, seed):
    rng = np.random.default_rng([int(seed), 77])
    made = ensemble_specimens(case, rng) if case["kind"] == "ensemble" else [SPECIMEN[case["kind"]](case, rng)]
    grad = rng.normal(size=(case["steps"], 2, 3)) if case["kind"] == "window" else None
    return made, grad


# ---------------------------------------------------------------------------
# the framework's side
# ---------------------------------------------------------------------------
def build(w, precision):
    sim = _capi.DemSim("RotSphere" if w["rot"] else "NRotSphere", w["grid"], w["skin"], w["lo"], w["hi"],
                       (1 if w["periodic"] else 0, 0, 0), w["dt"])
    n = len(w["rad"])
    sim.add_particles(np.arange(n, dtype=np.int32), w["pos"], w["rad"], sphere_mass(w["rad"]),
                      tag=np.zeros(n, np.int32), vel=w["vel"], angvel=w.get("angvel"))
    if "bonds" in w:
        i, j = w["bonds"]
        sim.add_connections(np.ones(len(i), np.int32), i, j)
        sim.add_rot_bond_group("bonds", 1, *w["bond_k"], *w["strength"], True, True, 1.0)
    if w["law"] == "elastic":
        sim.add_elastic_group("pairs", w["k"], True)
    elif w["law"] == "friction":
        sim.add_rot_friction_group("pairs", w["k"], w["mu"], w["mu"], w["ks"], w["dt"], True, True)
        if "bonds" in w:
            sim.add_exclusion("bonds", "pairs")
    elif w["law"] == "nfriction":
        sim.add_nrot_friction_group("pairs", w["k"], w["mu"], w["ks"], w["dt"], True)
    for name, o, nrm in w["walls"]:
        sim.add_wall(name, o, nrm)
        sim.add_wall_group(name + "_w", name, w["wall_k"])
    if "gravity" in w:
        sim.add_gravity("gravity", w["gravity"])
    for rot, visc, it in w.get("damping", ()):
        sim.add_damping(rot, visc, it)
    for name, v in w.get("wall_vel", {}).items():
        sim.set_wall_velocity(name, v)
    if precision != 64:
        sim.set_option("precision", precision)
    if "bonds" in w and w["law"]:
        sim.set_option("bond_handoff", 1)
    return sim


FIELDS = (("pos", 3), ("vel", 3), ("angvel", 3), ("quat", 4), ("force", 3), ("moment", 3))


def prepare(case, seed):
    made, grad = specimens(case, seed)
    sims = [build(w, case["precision"]) for w in made]
    n = sum(len(w["rad"]) for w in made)
    rot = made[0]["rot"]
    pin = torch.cuda.is_available()
    host = {k: torch.zeros((n, d), dtype=torch.float64, pin_memory=pin) for k, d in FIELDS
            if rot or k in ("pos", "vel", "force")}
    state = {"case": case, "sims": sims, "made": made, "host": host, "sizes": [len(w["rad"]) for w in made],
             "grad": grad}
    if case["kind"] == "ensemble":
        state["ensemble"] = _capi.Ensemble(sims)
    if case["kind"] == "window":
        sims[0].search_neighbors()
    return state


def read_back(state):
    """The state into the caller's pinned arrays, specimen after specimen, and the walls' reactions."""
    at, walls = 0, []
    for sim, n, w in zip(state["sims"], state["sizes"], state["made"]):
        ptr = [state["host"][k][at:].data_ptr() if k in state["host"] else 0 for k, _ in FIELDS]
        sim.get_particles_raw(0, *ptr)
        at += n
        for name, _, _ in w["walls"]:
            walls.append(np.stack(sim.wall(name)))
    return dict(state["host"], walls=np.stack(walls))


def run(state):
    case, sims = state["case"], state["sims"]
    kind = case["kind"]
    if kind == "window":
        sim = sims[0]
        reactions = sim.window_forward(case["steps"], case["every"])
        g = sim.window_adjoint(state["grad"])
        sim.window_rewind()
        return {"reactions": reactions, "params": g["params"], "pos": g["pos"], "vel": g["vel"],
                "angvel": g["angvel"], "quat": g["quat"]}
    if kind == "ensemble":
        state["ensemble"].step(case["steps"])
    elif kind == "flow":
        for _ in range(case["searches"]):
            sims[0].search_neighbors()
            sims[0].step(case["every"])
    else:
        sims[0].step(case["steps"])
        if state["made"][0].get("servo"):
            sims[0].apply_force_to_wall("top_w", state["made"][0]["servo"])
    return read_back(state)


def work(case):
    """Bytes and operations of a pass: each timestep reads and writes every particle's state once and reads every
    interaction once (tangential histories written too); a reverse step as two forward ones; the read-back."""
    kind = case["kind"]
    if kind == "gravity":
        n = case["side"] ** 2 * case["layers"]
    elif kind in ("pack", "flow"):
        n = case["nx"] * case["ny"] * case["nz"]
    elif kind == "ensemble":
        lo, hi = math.log(case["low"]), math.log(case["high"])
        n = case["specimens"] * (case["high"] - case["low"]) / (hi - lo) if hi > lo else case["specimens"] * case["high"]
    else:
        n = case["count"] * case.get("tx", 1) * case.get("ty", 1) * case.get("tz", 1)
    rot = kind not in ("gravity", "slide")
    steps = case["every"] * case["searches"] if kind == "flow" else case["steps"]
    # interactions per particle: list pairs, bonds
    pairs, bonds = {"gravity": (3.0, 0), "pack": (3.0, 0), "flow": (3.0, 0), "shear": (1.67, 0), "slide": (1.67, 0),
                    "block": (0.9, 3.7), "ensemble": (0.9, 3.6), "window": (0, 3.7)}[kind]
    history = 0 if kind == "gravity" else 2 * (16 if case["precision"] == 32 else 32)
    step = n * ((256 if rot else 136) + pairs * (8 + history) + bonds * (8 + 32))
    flops = n * ((150 if rot else 60) + pairs * (120 if kind != "gravity" else 25) + bonds * 600)
    if kind == "window":
        step, flops = 4 * step, 5 * flops  # forward, recompute and the reverse step's reads and writes
    out = n * (152 if rot else 72)
    searches = case["searches"] if kind == "flow" else 0
    return {"bytes": steps * step + out + searches * n * (64 + pairs * 32), "flops": steps * flops}


# ---------------------------------------------------------------------------
# the same physics in plain torch, 64 bits
# ---------------------------------------------------------------------------
def near_pairs(pos, rad, margin, length_x):
    """Pairs (i < j) within r_i + r_j + margin (periodic in x when length_x), by a cell grid."""
    n = len(rad)
    dev = pos.device
    c = 2 * float(rad.max()) + margin
    lo = pos.min(0).values - 1e-9
    dims = ((pos.max(0).values - lo) / c).floor().long() + 1
    size = torch.full((3,), c, dtype=torch.float64, device=dev)
    p = pos.clone()
    if length_x:
        nx = max(1, int(length_x // c))
        if nx < 3:
            raise ValueError("periodic box too small")
        dims[0], size[0], lo[0] = nx, length_x / nx, 0.0
        p[:, 0] = p[:, 0] % length_x
    q = ((p - lo) / size).floor().long()
    q = torch.minimum(q, dims - 1)
    key = (q[:, 0] * dims[1] + q[:, 1]) * dims[2] + q[:, 2]
    order = torch.argsort(key, stable=True)
    ncell = int(dims.prod())
    start = torch.searchsorted(key[order].contiguous(), torch.arange(ncell + 1, device=dev))
    found = []
    half = [(a, b, d) for a in (-1, 0, 1) for b in (-1, 0, 1) for d in (-1, 0, 1) if (a, b, d) >= (0, 0, 0)]
    for off in half:
        t = q + torch.tensor(off, device=dev)
        if length_x:
            t[:, 0] = t[:, 0] % dims[0]
        ok = ((t >= 0) & (t < dims)).all(1)
        i = torch.nonzero(ok)[:, 0]
        k = ((t[:, 0] * dims[1] + t[:, 1]) * dims[2] + t[:, 2])[i]
        count = start[k + 1] - start[k]
        a = torch.repeat_interleave(i, count)
        within = torch.arange(len(a), device=dev) - torch.repeat_interleave(torch.cumsum(count, 0) - count, count)
        b = order[torch.repeat_interleave(start[k], count) + within]
        if off == (0, 0, 0):
            keep = a < b
            a, b = a[keep], b[keep]
        d = pos[a] - pos[b]
        if length_x:
            d[:, 0] -= length_x * torch.round(d[:, 0] / length_x)
        near = (d * d).sum(1) <= (rad[a] + rad[b] + margin) ** 2
        a, b = a[near], b[near]
        found.append(torch.stack([torch.minimum(a, b), torch.maximum(a, b)]))
    ij = torch.cat(found, 1)
    return ij[:, torch.argsort(ij[0] * n + ij[1])]


def dot(a, b):
    return (a * b).sum(-1, keepdim=True)


def norm(a):
    return torch.sqrt(dot(a, a))


def cross(a, b):
    return torch.linalg.cross(a, b)


def quat_mul(a, b):
    s = a[:, :1] * b[:, :1] - dot(a[:, 1:], b[:, 1:])
    return torch.cat([s, a[:, :1] * b[:, 1:] + b[:, :1] * a[:, 1:] + cross(a[:, 1:], b[:, 1:])], 1)


def conj(q):
    return torch.cat([q[:, :1], -q[:, 1:]], 1)


def matrix(q):
    s, x, y, z = q.unbind(1)
    return torch.stack([torch.stack([s * s + x * x - y * y - z * z, 2 * (x * y + s * z), 2 * (x * z - s * y)], 1),
                        torch.stack([2 * (x * y - s * z), s * s - x * x + y * y - z * z, 2 * (y * z + s * x)], 1),
                        torch.stack([2 * (x * z + s * y), 2 * (y * z - s * x), s * s - x * x - y * y + z * z], 1)], 1)


def turn(m, v):
    return (m * v[:, None, :]).sum(2)


def turn_back(m, v):
    return (m * v[:, :, None]).sum(1)


def guarded(cond, value, other, fn):
    """fn(value) where cond, else `other`, with finite derivatives in both branches."""
    return torch.where(cond, fn(torch.where(cond, value, torch.full_like(value, 0.5))), torch.full_like(value, other))


class Exact:
    """One specimen stepped in torch: elastic, rotational-friction and translational-friction contacts, brittle
    elastic bonds (normal, shear, twist and bend springs), walls, gravity, viscous damping."""

    def __init__(self, w, device, grad=False):
        t = lambda a: torch.as_tensor(np.asarray(a, np.float64), device=device)  # noqa: E731
        self.w, self.dev, self.dt = w, device, w["dt"]
        self.x, self.v, self.r = t(w["pos"]).clone(), t(w["vel"]).clone(), t(w["rad"])[:, None]
        n = self.n = len(w["rad"])
        self.m = t(sphere_mass(w["rad"]))[:, None]
        self.rot = w["rot"]
        self.om = t(w["angvel"]).clone() if self.rot else torch.zeros(n, 3, dtype=torch.float64, device=device)
        self.I = 0.4 * self.m * self.r * self.r
        self.q = torch.zeros(n, 4, dtype=torch.float64, device=device)
        self.q[:, 0] = 1.0
        self.Lx = float(w["hi"][0] - w["lo"][0]) if w["periodic"] else 0.0
        self.walls = {name: [t(o).clone(), t(nrm)] for name, o, nrm in w["walls"]}
        self.reaction = {name: torch.zeros(3, dtype=torch.float64, device=device) for name in self.walls}
        self.old, self.due = self.x.clone(), False
        self.grad = grad
        self.visc = {rot: t(visc) for rot, visc, _ in w.get("damping", ())}
        if "bonds" in w:
            i, j = (torch.as_tensor(np.asarray(a), device=device) for a in w["bonds"])
            i, j = torch.minimum(i, j), torch.maximum(i, j)
            o = torch.argsort(i * n + j)
            self.b = torch.stack([i[o], j[o]])
            self.b_alive = torch.ones(len(i), 1, dtype=torch.bool, device=device)
            self.D0 = self.x[self.b[1]] - self.x[self.b[0]]
            self.bk = [t(k) for k in w["bond_k"]]
        if w["law"]:
            self.p = near_pairs(self.x, self.r[:, 0], 0.15, self.Lx)
            self.h = torch.zeros(self.p.shape[1], 3, dtype=torch.float64, device=device)
            self.slip = torch.zeros(self.p.shape[1], 1, dtype=torch.bool, device=device)
            if "bonds" in w:
                key, bkey = self.p[0] * n + self.p[1], self.b[0] * n + self.b[1]
                at = torch.searchsorted(bkey, key).clamp(max=len(bkey) - 1)
                self.held_by = torch.where(bkey[at] == key, at, torch.full_like(at, -1))

    def search(self):
        if self.Lx:
            lo = self.w["lo"][0]
            self.x[:, 0] -= self.Lx * torch.floor((self.x[:, 0] - lo) / self.Lx)
        self.old, self.due = self.x.clone(), False

    def contacts(self, F, M):
        w, i, j = self.w, self.p[0], self.p[1]
        if "bonds" in w:
            free = (self.held_by < 0) | ~self.b_alive[self.held_by.clamp(min=0), 0]
        D = self.x[i] - self.x[j]
        if self.Lx:
            D[:, 0] -= self.Lx * torch.round(D[:, 0] / self.Lx)
        eq = self.r[i] + self.r[j]
        touch = dot(D, D) < eq * eq
        if "bonds" in w:
            touch = touch & free[:, None]
        t = torch.nonzero(touch[:, 0])[:, 0]
        i, j, D, eq = i[t], j[t], D[t], eq[t]
        d = norm(D)
        R = 0.5 * eq
        if w["law"] == "nfriction":
            kn, ks = w["k"] * R, w["ks"] * R
        else:
            kn, ks = w["k"] * R * R / eq, (w["ks"] * R * R / eq if "ks" in w else None)
        fn = D * (kn * (d - eq) / d)  # on j
        F.index_add_(0, i, -fn)
        F.index_add_(0, j, fn)
        if w["law"] == "elastic":
            return
        arm_j = self.r[j] / eq * D
        arm_i = arm_j - D
        if w["law"] == "friction":
            ds = (self.v[j] + cross(self.om[j], arm_j) - self.v[i] - cross(self.om[i], arm_i)) * w["dt"]
        else:
            ds = (self.v[j] - self.v[i]) * w["dt"]
        ds = ds - dot(ds, D) / dot(D, D) * D
        h = self.h[t] + ks * ds
        size, limit = norm(h), norm(fn) * w["mu"]
        slip = size > limit
        h = torch.where(slip, h * (limit / torch.where(slip, size, torch.ones_like(size))), h)
        self.h = torch.zeros_like(self.h)
        self.h[t] = h
        F.index_add_(0, i, h)
        F.index_add_(0, j, -h)
        if w["law"] == "friction":
            M.index_add_(0, i, cross(arm_i, h))
            M.index_add_(0, j, cross(arm_j, -h))

    def bonds(self, F, M):
        w, i, j = self.w, self.b[0], self.b[1]
        kr, ks, kt, kb = self.bk
        mD = self.D0
        d0 = norm(mD)
        R = 0.5 * d0
        A, J = R * R, 0.5 * R ** 4
        kr, ks, kt, kb = kr * A / d0, ks * A / d0, kt * J / d0, kb * 0.5 * J / d0
        mn, ms, mt, mb = w["strength"]
        r1, r2 = self.r[i], self.r[j]
        r0 = r1 + r2
        q1 = self.q[i]
        m1 = matrix(q1)
        gap = self.x[j] - self.x[i]
        rb = turn(m1, gap)
        n = norm(rb)
        Fr = kr * (n - r0) * rb / n
        one = torch.ones_like(n)
        cg = dot(rb, mD) / (n * d0)
        gamma = guarded((cg < 1) & (cg > -1), cg, 0.0, torch.acos)
        c1 = cross(rb, mD)
        c2 = cross(rb, c1)
        has1, has2 = dot(c1, c1) != 0, dot(c2, c2) != 0
        n1 = torch.sqrt(torch.where(has1, dot(c1, c1), one))
        n2 = torch.sqrt(torch.where(has2, dot(c2, c2), one))
        Fst = torch.where(has2, ks * r0 * gamma * c2 / n2, torch.zeros_like(c2))
        fst2 = dot(Fst, Fst)
        some = fst2 != 0
        fst = torch.where(some, torch.sqrt(torch.where(some, fst2, one)), torch.zeros_like(fst2))
        Mst = torch.where(has1, -fst * c1 / n1, torch.zeros_like(c1))
        z = rb[:, 2:]
        h = math.sqrt(0.5)
        up, dn = (n + z) / n, (n - z) / n
        root = lambda a: torch.where(a > 0, torch.sqrt(torch.where(a > 0, a, one)), torch.zeros_like(a))  # noqa: E731
        m0, side = h * root(up), h * root(dn)
        xy = rb[:, :1] ** 2 + rb[:, 1:2] ** 2
        off = xy != 0
        sxy = torch.sqrt(torch.where(off, xy, one))
        mx = torch.where(off, -side * rb[:, 1:2] / sxy, -side)
        my = torch.where(off, side * rb[:, :1] / sxy, side)
        qm = torch.cat([m0, mx, my, torch.zeros_like(m0)], 1)
        mm = matrix(qm)
        r = quat_mul(quat_mul(conj(qm), quat_mul(conj(q1), self.q[j])), qm)
        s, a, b, c = (r[:, k:k + 1] for k in range(4))
        t0 = s * s + c * c
        cp, sp = s / torch.sqrt(t0), c / torch.sqrt(t0)
        ang = guarded((cp < 1) & (cp > -1), cp, 0.0, torch.acos)
        twist = 2 * torch.where(sp > 0, ang, torch.where(sp < 0, -ang, torch.zeros_like(ang)))
        zero = torch.zeros_like(twist)
        Mt = turn_back(mm, torch.cat([zero, zero, kt * twist], 1))
        t2 = a * a + b * b
        bent = t2 != 0
        t1 = t0 - t2
        sita = guarded(bent & (t1 < 1) & (t1 > -1), t1, 0.0, torch.acos)
        den = torch.sqrt(torch.where(bent, t0 * t2, one))
        cf = torch.where(bent, (a * c + s * b) / den, zero)
        sf = torch.where(bent, (b * c - s * a) / den, zero)
        Mb = turn_back(mm, torch.cat([-0.5 * kb * sita * sf, 0.5 * kb * sita * cf, zero], 1))
        g = 0.5 * ks * sita * r0
        Fs = turn_back(mm, torch.cat([-g * cf, -g * sf, zero], 1))
        Ms = turn_back(mm, torch.cat([g * sf, -g * cf, zero], 1))
        length = norm(gap)
        force = turn_back(m1, Fr + Fst + Fs)
        e1, e2 = r1 / r0 * length, r2 / r0 * length
        mo1 = turn_back(m1, Mb + Mt + (Ms + Mst) * e1)
        mo2 = turn_back(m1, (Ms + Mst) * e2 - Mb - Mt)
        on = self.b_alive.double()
        F.index_add_(0, i, force * on)
        F.index_add_(0, j, -force * on)
        M.index_add_(0, i, mo1 * on)
        M.index_add_(0, j, mo2 * on)
        if self.grad:
            return  # strengths far above the loads
        normal = torch.where(length < r0, -norm(Fr), norm(Fr)) / (mn * A) + norm(Mb) / (mb * 0.5 * J / R)
        shear = norm(Fst + Fs) / (ms * A) + norm(Mt) / (mt * J / R)
        self.broke = (normal > 1.0) | (shear > 1.0 - normal)

    def damp(self, rot, iters, v, F, mass):
        visc, s = self.visc[rot], 1.0 / mass
        rel, count = torch.zeros_like(v), torch.zeros_like(mass)
        go = torch.ones_like(mass, dtype=torch.bool)
        for _ in range(iters):
            new = v + s * self.dt * (F - rel * visc * mass)
            e = dot(new - rel, new - rel)
            rel = torch.where(go, new, rel)
            count = count + go
            go = go & (e * e > 1e-12)
            if not bool(go.any()):
                break
        rel = torch.where(count >= iters, torch.zeros_like(rel), rel)
        return F - visc * rel * mass

    def step(self):
        w, dt = self.w, self.dt
        if self.due:
            self.search()
        F = torch.zeros(self.n, 3, dtype=torch.float64, device=self.dev)
        M = torch.zeros_like(F)
        for name, (o, nrm) in self.walls.items():
            dist = dot(self.x - o, nrm)
            f = torch.where(dist < self.r, PI_REF * self.r * w["wall_k"] * (self.r - dist) * nrm, torch.zeros_like(F))
            F = F + f
            self.reaction[name] = f.sum(0)
        if "gravity" in w:
            F = F + torch.as_tensor(w["gravity"], dtype=torch.float64, device=self.dev) * self.m
        self.broke = None
        if w["law"]:
            self.contacts(F, M)
        if "bonds" in w:
            self.bonds(F, M)
        if self.broke is not None:
            self.b_alive = self.b_alive & ~self.broke
        for rot, _, it in w.get("damping", ()):
            if rot:
                M = self.damp(1, it, self.om, M, self.I)
            else:
                F = self.damp(0, it, self.v, F, self.m)
        if self.rot:
            self.om = self.om + dt / self.I * M
            dq = quat_mul(torch.cat([torch.zeros_like(self.m), self.om], 1), self.q)
            q = self.q + 0.5 * dt * dq
            self.q = q / norm(q)
        self.v = self.v + F / self.m * dt
        self.x = self.x + self.v * dt
        self.F, self.M = F, M
        if not self.grad:
            moved = ((self.x - self.old) ** 2).sum(1)
            self.due = bool((moved > (0.5 * w["skin"]) ** 2).any())
        for name, v in w.get("wall_vel", {}).items():
            o, nrm = self.walls[name]
            self.walls[name] = [o + torch.as_tensor(v, dtype=torch.float64, device=self.dev) * dt, nrm]

    def servo(self, name, force):
        """Moves a wall along `force` until its spheres carry it."""
        f = torch.as_tensor(force, dtype=torch.float64, device=self.dev)
        size = float(f.norm())
        u = f / size
        o, nrm = self.walls[name]
        for _ in range(50):
            dist = dot(self.x - o, nrm)
            touch = dist < self.r
            k = PI_REF * self.r * self.w["wall_k"] * touch
            K = float(k.sum())
            if K > 0:
                push = -(k * (self.r - dist) * nrm).sum(0)
                df = float((f + (push * u).sum() * u) @ u)
                move, off = df / K, df / size
            else:
                move, off = 1e-5, 1.0
            o = o + move * u
            if not off > 1e-3:
                break
        self.walls[name] = [o, nrm]


def exact(case, seed):
    made, grad = specimens(case, seed)
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    if case["kind"] == "window":
        return exact_window(case, made[0], grad, dev)
    host, walls = {k: [] for k, _ in FIELDS}, []
    for w in made:
        e = Exact(w, dev)
        if case["kind"] == "flow":
            for _ in range(case["searches"]):
                e.search()
                for _ in range(case["every"]):
                    e.step()
        else:
            for _ in range(case["steps"]):
                e.step()
            if w.get("servo"):
                e.servo("top", w["servo"])
        for k, v in zip(("pos", "vel", "angvel", "quat", "force", "moment"), (e.x, e.v, e.om, e.q, e.F, e.M)):
            host[k].append(v.cpu())
        for name, _, _ in w["walls"]:
            walls.append(torch.stack([e.walls[name][0], e.reaction[name]]).cpu().numpy())
    rot = made[0]["rot"]
    out = {k: torch.cat(v) for k, v in host.items() if rot or k in ("pos", "vel", "force")}
    return dict(out, walls=np.stack(walls))


def exact_window(case, w, grad, dev):
    e = Exact(w, dev, grad=True)
    leaves = [e.x, e.v, e.om, e.q] + e.bk + [e.visc[0], e.visc[1]]
    for a in leaves:
        a.requires_grad_(True)
    g = torch.as_tensor(grad, device=dev)
    loss, reactions = 0.0, []
    for k in range(case["steps"]):
        e.step()
        r = torch.stack([e.reaction["bottom"], e.reaction["top"]])
        loss = loss + (r * g[k]).sum()
        reactions.append(r.detach())
    d = torch.autograd.grad(loss, leaves)
    # the bonds start at rest, where the angle acos(c) of a bond has no derivative (c rounds to 1 or to just below):
    # gradients with respect to the initial positions and orientations, which pass through it, have no value
    return {"reactions": torch.stack(reactions).cpu().numpy(), "params": torch.stack(list(d[4:])).cpu().numpy(),
            "vel": d[1].cpu().numpy(), "angvel": d[2].cpu().numpy(), "pos": None, "quat": None}
