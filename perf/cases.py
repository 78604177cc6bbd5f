"""Workloads of the DEM engine that are timed and compared between two builds.

Each case is what a user of the framework runs through nbc.py: an engine that
is stepped and read back, a batch of scenes, a request server, a cell sort on
the caller's own buffers.  The beds come from the repository's settled states
(50,000 tetrahedral clumps in a cylinder after 20,000 steps, 2,000 spheres in
a box after 10,000), turned, cropped and tiled to the size asked for, so that
they carry the contacts, the wall contacts and the rebuild rate of a real run;
the polydisperse beds are freshly seeded and falling, the first phase of every
penetration test.

`exact` is an FP64 restatement of the step in torch that shares nothing with
the engine: its own pair search, its own sums.
"""
import math
import os
import random
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, os.path.join(ROOT, "nbody-clump_b200"))
import nbc  # noqa: E402
import scenegen  # noqa: E402

GOLDEN = os.path.join(ROOT, "tests", "golden")
BED_R = 0.06          # radius of the settled bed of clumps
TILE = 0.0418         # half side of the square column cut from it
SPHERE_BOX = 0.04     # side of the settled box of spheres


def listed():
    return [
        # the smallest calls: a correctness-sized scene in the reference's own
        # precision, and the smallest scene a batch or a request holds
        {"name": "spheres_2k_f64", "kind": "spheres", "n": 2000, "law": "f64", "driver": "clump", "mu": 0.5,
         "steps": 400},
        {"name": "clumps_500", "kind": "clumps", "n": 500, "law": "mixed", "wall": "cylinder", "mu": 0.35,
         "intruder_mm": 0.0, "speed": 0.0, "rows": 128, "steps": 400},
        # ordinary scenes: the sphere-only cube driver at an odd size, a few
        # thousand clumps, a penetration test in a box (its force-depth curve
        # is the result), a scene in FP64 at an odd size
        {"name": "spheres_driver_9k_f64", "kind": "spheres", "n": 9217, "law": "f64", "driver": "cube", "mu": 0.5,
         "steps": 300},
        {"name": "clumps_5k", "kind": "clumps", "n": 5000, "law": "mixed", "wall": "cylinder", "mu": 0.6,
         "intruder_mm": 0.0, "speed": 0.0, "rows": 0, "steps": 300},
        {"name": "penetration_12k", "kind": "clumps", "n": 12007, "law": "mixed", "wall": "cube", "mu": 0.5,
         "intruder_mm": 12.0, "speed": 0.3, "rows": 0, "steps": 250},
        {"name": "clumps_13k_f64", "kind": "clumps", "n": 13331, "law": "f64", "wall": "cylinder", "mu": 0.5,
         "intruder_mm": 0.0, "speed": 0.0, "rows": 0, "steps": 250},
        # the benchmark's scene, and the largest: a million subspheres in a box
        {"name": "clumps_50k", "kind": "clumps", "n": 50000, "law": "mixed", "wall": "cylinder", "mu": 0.5,
         "intruder_mm": 0.0, "speed": 0.0, "rows": 0, "steps": 200},
        {"name": "clumps_250k", "kind": "clumps", "n": 250000, "law": "mixed", "wall": "cube", "mu": 0.5,
         "intruder_mm": 0.0, "speed": 0.0, "rows": 0, "steps": 60},
        # a polydisperse bed falling into place: radii 0.5 to 5 mm, clumps of
        # one to eight subspheres, the hierarchical grid
        {"name": "poly_fall_60k", "kind": "poly", "n": 60000, "law": "mixed", "mu": 0.5, "fall": 0.9, "steps": 200},
        # many scenes of uneven size in one engine, and requests served
        # together from submission to their force curves
        {"name": "batch_24", "kind": "batch", "scenes": 24, "low": 500, "high": 8000, "law": "mixed", "steps": 200},
        {"name": "serve_8", "kind": "serve", "scenes": 8, "low": 300, "high": 5000, "law": "mixed", "steps": 400},
        # the cell sort on a caller's own buffers
        {"name": "cell_sort_180k", "kind": "sort", "n": 180001, "edge": 48},
    ]


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["spheres"] * 2 + ["clumps"] * 4 + ["penetration", "penetration", "poly", "batch", "serve", "sort"])
    mu = round(rng.uniform(0.2, 0.8), 3)
    law = rng.choice(["mixed", "mixed", "mixed", "f64"])
    if kind == "spheres":
        n = _log_uniform(rng, 700, 60000)
        return {"kind": "spheres", "n": n, "law": rng.choice(["f64", "mixed"]), "driver": rng.choice(["clump", "cube"]),
                "mu": mu, "steps": 300}
    if kind in ("clumps", "penetration"):
        n = _log_uniform(rng, 400, 150000 if law == "mixed" else 40000)
        pene = kind == "penetration"
        wall = "cube" if pene or n > 30000 else rng.choice(["cylinder", "cube"])
        return {"kind": "clumps", "n": n, "law": law, "wall": wall, "mu": mu,
                "intruder_mm": round(rng.uniform(5, 20), 2) if pene else 0.0,
                "speed": round(rng.uniform(0.05, 0.5), 3) if pene else 0.0,
                "rows": 128 if n < 1500 else 0, "steps": 300 if n < 10000 else (200 if n < 60000 else 80)}
    if kind == "poly":
        return {"kind": "poly", "n": _log_uniform(rng, 3000, 60000), "law": law, "mu": mu,
                "fall": round(rng.uniform(0.3, 1.5), 3), "steps": 200}
    if kind == "batch":
        return {"kind": "batch", "scenes": rng.randint(3, 24), "low": 500, "high": _log_uniform(rng, 1000, 8000),
                "law": "mixed", "steps": 200}
    if kind == "serve":
        return {"kind": "serve", "scenes": rng.randint(2, 8), "low": 250, "high": _log_uniform(rng, 800, 5000),
                "law": "mixed", "steps": rng.choice([200, 300, 400])}
    return {"kind": "sort", "n": _log_uniform(rng, 1500, 262144), "edge": rng.randint(9, 100)}


# ---------------------------------------------------------------------------
# scenes
# ---------------------------------------------------------------------------

_beds = {}


def _settled_clumps():
    """The repository's settled bed of clumps (read once; the same for every seed)."""
    if "clumps" not in _beds:
        s = scenegen.tetra_state_from_npz(os.path.join(GOLDEN, "cfg1_settled.npz"))
        k = s["params"]["ClumpNum"]
        _beds["clumps"] = {
            "params": s["params"], "pos": s["clump"]["pos"], "quat": s["clump"]["quat"], "vel": s["clump"]["vel"],
            "angvel": s["clump"]["angvel"], "prop": s["clump"]["prop"], "spos": s["sub"]["pos"].reshape(k, 4, 3),
            "local": s["sub"]["local"].reshape(k, 4, 3), "radius": s["sub"]["radius"].reshape(k, 4),
            "mass": s["sub"]["mass"].reshape(k, 4)}
    return _beds["clumps"]


def _settled_spheres():
    if "spheres" not in _beds:
        z = np.load(os.path.join(GOLDEN, "cfg0_settle.ref.npz"))
        _beds["spheres"] = {k: z["s10000/clump_" + k] for k in ("pos", "vel", "quat", "angvel")}
    return _beds["spheres"]


def _turn(v, c, s):
    """Rotation about z of the vectors v by the angle with this cosine and sine."""
    o = v.copy()
    o[..., 0], o[..., 1] = c * v[..., 0] - s * v[..., 1], s * v[..., 0] + c * v[..., 1]
    return o


def _turn_quat(q, a):
    """The attitudes q (x y z w) turned by the angle a about the world z axis."""
    s, c = math.sin(0.5 * a), math.cos(0.5 * a)
    return np.stack([c * q[:, 0] - s * q[:, 1], c * q[:, 1] + s * q[:, 0], c * q[:, 2] + s * q[:, 3],
                     c * q[:, 3] - s * q[:, 2]], axis=1)


def _turned(bed, a, shift=(0.0, 0.0)):
    c, s = math.cos(a), math.sin(a)
    off = np.array([shift[0], shift[1], 0.0])
    return {"pos": _turn(bed["pos"], c, s) + off, "vel": _turn(bed["vel"], c, s), "angvel": _turn(bed["angvel"], c, s),
            "quat": _turn_quat(bed["quat"], a), "spos": _turn(bed["spos"], c, s) + off}


def _clump_scene(n, seed, wall, mu):
    """n clumps of the settled bed, the lowest ones of a column cut from it
    (several columns side by side for the large sizes), in a wall of that
    size; the bed is turned by an angle of the seed first."""
    bed = _settled_clumps()
    rng = np.random.default_rng(seed)
    angle = rng.uniform(0, 2 * math.pi)
    rad, K0 = bed["radius"], len(bed["pos"])
    parts = []
    if wall == "cylinder":
        size = BED_R * (n / K0) ** (1 / 3)
        t = _turned(bed, angle)
        reach = (np.hypot(t["spos"][..., 0], t["spos"][..., 1]) + rad).max(1)
        while True:
            keep = np.nonzero(reach <= size)[0] if size < BED_R else np.arange(K0)
            if len(keep) >= n or size >= BED_R:
                break
            size *= 1.03
        size = min(size, BED_R)
        parts.append((t, keep))
        half = (size, size)
    else:
        full = int(0.55 * K0)   # a square column holds more than this
        m = max(1, math.ceil(math.sqrt(n / full)))
        size = TILE * min(1.0, (n / full) ** (1 / 3))
        while True:
            parts = []
            for i in range(m * m):
                t = _turned(bed, angle + 2 * math.pi * i / (m * m))
                reach = np.maximum(np.abs(t["spos"][..., 0]), np.abs(t["spos"][..., 1])) + rad
                keep = np.nonzero(reach.max(1) <= size)[0]
                off = ((i % m - 0.5 * (m - 1)) * 2 * size, (i // m - 0.5 * (m - 1)) * 2 * size, 0.0)
                t["pos"] = t["pos"] + np.array(off)
                t["spos"] = t["spos"] + np.array(off)
                parts.append((t, keep))
            if sum(len(k) for _, k in parts) >= n or size >= TILE:
                break
            size = min(TILE, size * 1.03)
        half = (m * size, m * size)
    pick = {k: np.concatenate([t[k][keep] for t, keep in parts]) for k in ("pos", "vel", "angvel", "quat", "spos")}
    pick.update({k: np.concatenate([bed[k][keep] for _, keep in parts]) for k in ("prop", "local", "radius", "mass")})
    low = np.sort(np.argsort(pick["pos"][:, 2], kind="stable")[:n])
    pick = {k: v[low] for k, v in pick.items()}
    k = len(low)
    pick["vel"] = pick["vel"] + rng.normal(0, 1e-3, (k, 3))
    params = dict(bed["params"], NumberBody=4 * k, ClumpNum=k, Frcoe=float(mu))
    top = float((pick["spos"][..., 2] + pick["radius"]).max())
    scenegen.set_world_box(params, (-half[0], -half[1], 0.0), (half[0], half[1], min(0.3, 1.25 * top)))
    scene = {"params": params,
             "sub": {"clump_id": np.repeat(np.arange(k, dtype=np.int32), 4), "pos": pick["spos"].reshape(-1, 3),
                     "local": pick["local"].reshape(-1, 3), "mass": pick["mass"].reshape(-1),
                     "radius": pick["radius"].reshape(-1)},
             "clump": {c: np.ascontiguousarray(pick[c]) for c in ("pos", "vel", "quat", "angvel", "prop")},
             "cube": None, "cylinder": None, "intruder": None}
    if wall == "cylinder":
        scene["cylinder"] = scenegen.make_cylinder(half[0], 0.15, (0, 0, 0.15))
    else:
        scene["cube"] = scenegen.make_cube((half[0], half[1], 0.15), (0, 0, 0.15))
    return nbc.with_levels(scene)


def _sphere_scene(n, seed, driver, mu):
    """n spheres of the settled box, mirrored and turned by the seed, several
    boxes side by side for the larger sizes, the lowest n kept."""
    bed = _settled_spheres()
    rng = np.random.default_rng(seed)
    m = max(1, math.ceil(math.sqrt(n / len(bed["pos"]))))
    mid = np.array([0.5 * SPHERE_BOX, 0.5 * SPHERE_BOX, 0.0])
    pos, vel, quat, wel = [], [], [], []
    for i in range(m * m):
        a = 0.5 * math.pi * int(rng.integers(0, 4))
        c, s = round(math.cos(a)), round(math.sin(a))
        p = _turn(bed["pos"] - mid, c, s) + mid
        pos.append(p + np.array([(i % m) * SPHERE_BOX, (i // m) * SPHERE_BOX, 0.0]))
        vel.append(_turn(bed["vel"], c, s))
        wel.append(_turn(bed["angvel"], c, s))
        quat.append(_turn_quat(bed["quat"], a))
    pos, vel, quat, wel = (np.concatenate(v) for v in (pos, vel, quat, wel))
    low = np.sort(np.argsort(pos[:, 2], kind="stable")[:n])
    pos, vel, quat, wel = pos[low], vel[low], quat[low], wel[low]
    vel = vel + rng.normal(0, 5e-3, vel.shape)
    r, rho = 1e-3, scenegen.MATERIAL["rho"]
    mass = rho * 4 / 3 * math.pi * r ** 3
    inertia = 0.4 * mass * r * r
    M = scenegen.MATERIAL
    params = scenegen.default_params(StepSize=0.2 * scenegen.rayleigh_dt(r, rho, M["Ymod"], M["Prat"]), Ymod=M["Ymod"],
                                     Prat=M["Prat"], Frcoe=float(mu), NormRes=M["NormRes"], Thresh=0.2 * r,
                                     BranchLmtLen=64, NumberBody=n, ClumpNum=n)
    side = m * SPHERE_BOX
    scenegen.set_world_box(params, (0, 0, 0), (side, side, 0.08))
    scene = {"params": params,
             "sub": {"clump_id": np.arange(n, dtype=np.int32), "pos": pos.copy(), "local": np.zeros((n, 3)),
                     "mass": np.full(n, mass), "radius": np.full(n, r)},
             "clump": {"pos": pos, "vel": vel, "quat": quat, "angvel": wel,
                       "prop": np.tile([inertia, inertia, inertia, mass], (n, 1))},
             "cube": scenegen.make_cube((0.5 * side, 0.5 * side, 0.04), (0.5 * side, 0.5 * side, 0.04)),
             "cylinder": None, "intruder": None}
    return scenegen.as_sphere_driver(scene, "cube") if driver == "cube" else scene


def _poly_scene(n, seed, mu, fall):
    """A seeded polydisperse bed that has fallen to the speed `fall`."""
    scene = scenegen.make_poly_bed(n, seed, 0.2 * (n / 1e6) ** (1 / 3), mu=mu)
    rng = np.random.default_rng(seed + 1)
    k = len(scene["clump"]["vel"])
    scene["clump"]["vel"] = rng.normal(0, 0.1 * fall, (k, 3)) + np.array([0.0, 0.0, -fall])
    scene["clump"]["angvel"] = rng.normal(0, 20.0, (k, 3))
    return nbc.with_levels(scene)


def _uneven(case, seed):
    """The scenes of a batch, or of the requests of a server: clump counts
    log-uniform (the case's), friction and state the seed's."""
    sizes, rng = random.Random(case["scenes"]), random.Random(seed)
    out = []
    for i in range(case["scenes"]):
        n = _log_uniform(sizes, case["low"], case["high"])
        wall = "cube" if case["kind"] == "serve" else "cylinder"
        sc = _clump_scene(n, seed + 17 * i, wall, rng.uniform(0.2, 0.8))
        if case["kind"] == "serve":
            sc = scenegen.with_sphere_intruder(sc, rng.uniform(5e-3, 12e-3), rng.uniform(0.05, 0.5), surface=98)
        out.append(sc)
    return out


def _request_steps(case):
    """The step counts of a server's requests: uneven, the longest is case["steps"]."""
    return [case["steps"] - 50 * (i % 3) for i in range(case["scenes"])]


def _scene(case, seed):
    if case["kind"] == "spheres":
        return _sphere_scene(case["n"], seed, case["driver"], case["mu"])
    if case["kind"] == "poly":
        return _poly_scene(case["n"], seed, case["mu"], case["fall"])
    sc = _clump_scene(case["n"], seed, case["wall"], case["mu"])
    if case["intruder_mm"] > 0:
        sc = scenegen.with_sphere_intruder(sc, 1e-3 * case["intruder_mm"], case["speed"], surface=98)
    return sc


# ---------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------

def prepare(case, seed):
    """What a user's program holds before the call: an engine made from its
    scene (or a batch, or a server and its scenes), or the buffers to sort."""
    if case["kind"] == "sort":
        n, e = case["n"], case["edge"]
        g = torch.Generator(device="cuda").manual_seed(int(seed))
        cell = 3e-3
        pos = torch.rand(n, 3, dtype=torch.float64, device="cuda", generator=g) * (cell * e)
        pos[:, 2] *= 0.7        # the upper part of the box is empty
        pos[: n // 997] += 1.0  # a few have left it
        grid = nbc.GridDesc()
        for a in range(3):
            grid.origin[a], grid.dims[a] = -cell, e + 2
            grid.box_lo[a], grid.box_hi[a] = 0.0, cell * e
        grid.cell = cell
        return {"case": case, "pos": pos, "grid": grid,
                "perm": torch.empty(n, dtype=torch.int32, device="cuda"),
                "key": torch.empty(n, dtype=torch.int32, device="cuda")}
    if case["kind"] == "batch":
        return {"case": case, "batch": nbc.Batch(_uneven(case, seed), precision=case["law"])}
    if case["kind"] == "serve":
        return {"case": case, "scenes": _uneven(case, seed),
                "server": nbc.Server(budget_bytes=20e9, max_active=64, precision=case["law"])}
    return {"case": case, "engine": nbc.Engine([_scene(case, seed)], precision=case["law"])}


def run(state):
    case = state["case"]
    if case["kind"] == "sort":
        nbc.cell_sort_noalloc(state["pos"].data_ptr(), case["n"], state["grid"], state["perm"].data_ptr(),
                              state["key"].data_ptr(), torch.cuda.current_stream().cuda_stream)
        return {"perm": state["perm"], "key": state["key"]}
    if case["kind"] == "batch":
        b = state["batch"]
        b.step(case["steps"])
        b.sync()
        got = [v.clumps() for v in b.engines]
        stats = [v.stats() for v in b.engines]
        out = {k: np.concatenate([g[k] for g in got]) for k in got[0]}
        out["stats"] = np.array([[s["steps"], s["rebuilds"], s["npairs"]] for s in stats])
        return out
    if case["kind"] == "serve":
        s = state["server"]
        ids = [s.submit(sc, n, sample_every=50) for sc, n in zip(state["scenes"], _request_steps(case))]
        while True:
            a = s.advance(200)
            if a["running"] == 0 and a["queued"] == 0:
                break
        got = [s.result(i) for i in ids]
        for i in ids:
            s.release(i)
        return {"curve": np.concatenate([g["curve"] for g in got]), "pos": np.array([g["intr_pos"] for g in got]),
                "steps": np.array([g["steps"] for g in got])}
    e = state["engine"]
    e.step(case["steps"])
    e.sync()
    out = e.clumps(0)
    s = e.stats(0)
    out["stats"] = np.array([s["steps"], s["rebuilds"], s["npairs"]])
    if case.get("rows"):
        out["rows"], out["front"], out["back"] = e.rows(0, case["rows"])
    if case.get("intruder_mm"):
        out["curve"] = e.intruder_history(0, case["steps"])
    return out


def work(case):
    """Per step and clump: pose, velocities in and out, inertia in; per
    subsphere: its offset, mass and radius in; per contact (about half of one
    per subsphere of a clump bed, two per sphere, few in a falling bed): two
    indices and its springs in and out."""
    if case["kind"] == "sort":
        return {"bytes": 32.0 * case["n"], "flops": 10.0 * case["n"]}
    if case["kind"] in ("batch", "serve"):
        lo, hi = case["low"], case["high"]
        k = case["scenes"] * (hi - lo) / math.log(hi / lo)
        n, contacts = 4.0 * k, 2.0 * k
    elif case["kind"] == "clumps":
        k, n, contacts = case["n"], 4.0 * case["n"], 2.0 * case["n"]
    elif case["kind"] == "spheres":
        k, n, contacts = case["n"], case["n"], 2.0 * case["n"]
    else:
        k, n, contacts = case["n"] / 4.5, case["n"], 0.05 * case["n"]
    word = 8 if case["law"] == "f64" else 4
    return {"bytes": case["steps"] * (k * (2 * 104 + 32) + n * 40 + contacts * (8 + 2 * 9 * word)),
            "flops": case["steps"] * (k * 250.0 + n * 60.0 + contacts * 300.0)}


# ---------------------------------------------------------------------------
# the step in 64 bits
# ---------------------------------------------------------------------------

def _dot(a, b):
    return (a * b).sum(-1, keepdim=True)


def _len(a):
    t = _dot(a, a)
    return torch.where(t > 1e-32, t.clamp_min(1e-300).sqrt(), torch.zeros_like(t))


def _cross(a, b):
    return torch.linalg.cross(a, b, dim=-1)


def _matrix(q):
    """Body-to-world rotation of the attitudes q (x y z w), not normalised."""
    x, y, z, w = q.unbind(-1)
    return torch.stack([
        torch.stack([x * x - y * y - z * z + w * w, 2 * (x * y - z * w), 2 * (x * z + y * w)], -1),
        torch.stack([2 * (x * y + z * w), -x * x + y * y - z * z + w * w, 2 * (y * z - x * w)], -1),
        torch.stack([2 * (x * z - y * w), 2 * (y * z + x * w), -x * x - y * y + z * z + w * w], -1)], -2)


def _half_rate(W, q):
    x, y, z, w = q.unbind(-1)
    a, b, c = W.unbind(-1)
    return 0.5 * torch.stack([a * w - b * z + c * y, a * z + b * w - c * x, -a * y + b * x + c * w,
                              -a * x - b * y - c * z], -1)


class _Exact:
    def __init__(self, scene, device):
        def t(a):
            return torch.as_tensor(np.ascontiguousarray(a), dtype=torch.float64, device=device)
        p, s, c = scene["params"], scene["sub"], scene["clump"]
        self.dev = device
        self.dt, self.g, self.mu, self.beta = p["StepSize"], p["Gravity"], p["Frcoe"], p["Beta"]
        self.kn = 2 * p["Ymod"] / (3 * (1 - p["Prat"] ** 2))
        self.ks = 2 * p["Ymod"] / (1 + p["Prat"]) / (2 - p["Prat"])
        ln, pi = math.log(p["NormRes"]), 3.14159265359
        self.damp = 2 * math.sqrt(5 / 6) * ln / math.sqrt(ln * ln + pi * pi)
        self.cid = torch.as_tensor(np.asarray(s["clump_id"], np.int64), device=device)
        self.r, self.m, self.local = t(s["radius"])[:, None], t(s["mass"])[:, None], t(s["local"])
        self.X, self.V, self.Q, self.W = t(c["pos"]), t(c["vel"]), t(c["quat"]), t(c["angvel"])
        prop = t(c["prop"])
        self.I, self.M = prop[:, :3], prop[:, 3:]
        self.F, self.T = torch.zeros_like(self.X), torch.zeros_like(self.X)
        self.n = len(self.cid)
        self.margin = 0.25 * float(self.r.min())
        self.at = None
        self.near = None
        self.held = None    # (keys, tangential, rolling, twisting springs) of the touching pairs
        self.wall_held = {}
        self.cube, self.cyl = scene.get("cube"), scene.get("cylinder")
        self.memory = not (scene.get("sphere_mode", 0) & nbc.SPHERE_CUBE_WALL)
        it = scene.get("intruder")
        self.intr = None
        if it is not None:
            self.intr = {"R": it["radius"], "p": t(it["pos"]).clone(), "v": t(it["vel"])}
        self.record = []

    def law(self, n, dn, vtot, dth, rij, mij, cs_mult, hs, hr, ht):
        sq = (rij * dn).sqrt()
        kn = self.kn * sq
        cn = self.damp * (kn * mij).sqrt()
        ks = self.ks * sq
        cs = cs_mult * self.damp * (ks * mij).sqrt()
        br2 = (self.beta * rij) ** 2
        kr, cr, kt, ct = 0.25 * kn * br2, 0.25 * cn * br2, 0.5 * ks * br2, 0.5 * cs * br2
        vn = _dot(n, vtot) * n
        vt = vtot - vn
        fn = kn * dn * n + cn * vn
        fl = _len(fn)

        def cap(v, limit, rest):
            l = _len(v)
            over = l > limit
            cut = torch.where(over, limit / torch.where(over, l, torch.ones_like(l)), torch.ones_like(l)) * v
            return torch.where(over, cut, v + rest), torch.where(over, cut, v), over
        ft = -ks * (self.dt * vt) + cs * vt + hs
        l = _len(ft)
        over = l > fl * self.mu
        ft = torch.where(over, self.mu * fl / torch.where(over, l, torch.ones_like(l)) * ft, ft)
        hs = torch.where(over, ft, ft - cs * vt)
        dt_ = _dot(dth, n) * n
        dr = dth - dt_
        mr, hr, _ = cap(kr * dr + hr, 0.525 * self.beta * rij * fl, -cr / self.dt * dr)
        mt, ht, _ = cap(kt * dt_ + ht, 0.65 * self.mu * self.beta * rij * fl, -ct / self.dt * dt_)
        return fn, ft, mr, mt, hs, hr, ht

    def search(self, p):
        """Pairs of different clumps closer than ri + rj + 2 margin."""
        cell = float(2 * self.r.max() + 2 * self.margin)
        c = torch.floor((p - p.min(0).values) / cell).long() + 1
        dims = (c.max(0).values + 2).tolist()
        key = (c[:, 2] * dims[1] + c[:, 1]) * dims[0] + c[:, 0]
        key, order = torch.sort(key, stable=True)
        steps = [(dz * dims[1] + dy) * dims[0] + dx for dz in (-1, 0, 1) for dy in (-1, 0, 1) for dx in (-1, 0, 1)]
        found = []
        me = torch.arange(self.n, device=self.dev)
        for s in steps:
            if s < 0:
                continue
            lo = torch.searchsorted(key, key + s) if s else me + 1
            cnt = (torch.searchsorted(key, key + s, right=True) - lo).clamp_min(0)
            a = torch.repeat_interleave(me, cnt)
            first = torch.cumsum(cnt, 0) - cnt
            b = lo[a] + (torch.arange(len(a), device=self.dev) - first[a])
            i, j = order[a], order[b]
            reach = self.r[i, 0] + self.r[j, 0] + 2 * self.margin
            ok = (((p[i] - p[j]) ** 2).sum(1) < reach * reach) & (self.cid[i] != self.cid[j])
            i, j = i[ok], j[ok]
            found.append(torch.stack([torch.minimum(i, j), torch.maximum(i, j)]))
        i, j = torch.cat(found, 1)
        k, o = torch.sort(i * self.n + j)
        self.near = (i[o], j[o], k)
        self.at = p.clone()

    def springs(self, keys, held):
        """The springs of the contacts `keys` (ascending), zero for those not held."""
        out = [torch.zeros(len(keys), 3, dtype=torch.float64, device=self.dev) for _ in range(3)]
        if held is not None and len(held[0]):
            at = torch.searchsorted(held[0], keys).clamp_max(len(held[0]) - 1)
            same = held[0][at] == keys
            for o, h in zip(out, held[1:]):
                o[same] = h[at[same]]
        return out

    def step(self):
        dt = self.dt
        down = torch.tensor([0.0, 0.0, self.g], dtype=torch.float64, device=self.dev)
        acc, al = self.F / self.M + down, self.T / self.I
        self.X = self.X + dt * self.V + 0.5 * dt * dt * acc
        self.V = self.V + 0.5 * dt * acc
        self.W = self.W + 0.5 * dt * al
        Rt = _matrix(self.Q).transpose(-1, -2)
        Wb, Ab = (Rt @ self.W[..., None])[..., 0], (Rt @ al[..., None])[..., 0]
        qd = _half_rate(Wb, self.Q)
        qdd = _half_rate(Ab, self.Q) + _half_rate(Wb, qd)
        q = self.Q + dt * qd + 0.5 * dt * dt * qdd
        self.Q = q / q.norm(dim=-1, keepdim=True)
        if self.intr is not None:
            self.intr["p"] = self.intr["p"] + dt * self.intr["v"]
        arm = (_matrix(self.Q)[self.cid] @ self.local[..., None])[..., 0]
        p = self.X[self.cid] + arm
        if self.at is None or float(((p - self.at) ** 2).sum(1).max()) > (0.99 * self.margin) ** 2:
            self.search(p)
        f, t = torch.zeros_like(p), torch.zeros_like(p)
        v, w = self.V[self.cid], self.W[self.cid]
        self.pairs(p, arm, v, w, f, t)
        self.walls(p, arm, v, w, f, t)
        if self.intr is not None:
            self.intruder(p, arm, v, w, f, t)
        t = t + _cross(p - self.X[self.cid], f)
        self.F = torch.zeros_like(self.X).index_add_(0, self.cid, f)
        self.T = torch.zeros_like(self.X).index_add_(0, self.cid, t)
        self.V = self.V + 0.5 * dt * (self.F / self.M + down)
        self.W = self.W + 0.5 * dt * (self.T / self.I)

    def pairs(self, p, arm, v, w, f, t):
        i, j, key = self.near
        d = p[j] - p[i]
        dist = d.norm(dim=1, keepdim=True)
        on = (self.r[i] + self.r[j] - dist > 0)[:, 0]
        i, j, key, d, dist = i[on], j[on], key[on], d[on], dist[on]
        ri, rj = self.r[i], self.r[j]
        n = d / dist
        ap = 0.5 * (ri * ri - rj * rj + dist * dist) / dist
        an = dist - ap
        ab = 0.5 * (rj * rj - ri * ri + dist * dist) / dist
        vtot = v[j] - v[i] + _cross(w[j], arm[j] - an * n) - _cross(w[i], arm[i] + ap * n)
        hs, hr, ht = self.springs(key, self.held)
        fn, ft, mr, mt, hs, hr, ht = self.law(n, ri + rj - dist, vtot, self.dt * (w[i] - w[j]), ri * rj / (ri + rj),
                                              self.m[i] * self.m[j] / (self.m[i] + self.m[j]), 1.0, hs, hr, ht)
        self.held = (key, hs, hr, ht)
        nxf = _cross(n, ft)
        f.index_add_(0, i, -fn - ft)
        f.index_add_(0, j, fn + ft)
        t.index_add_(0, i, -ap * nxf - mr - mt)
        t.index_add_(0, j, -ab * nxf + mr + mt)

    def one_sided(self, slot, i, n, ap, dn, arm, v, w, f, t, vw, rij, mij, cs, memory=True):
        hs, hr, ht = self.springs(i, self.wall_held.get(slot) if memory else None)
        vtot = v[i] - vw + _cross(-arm[i] + ap * n, w[i])
        fn, ft, mr, mt, hs, hr, ht = self.law(n, dn, vtot, self.dt * w[i], rij, mij, cs, hs, hr, ht)
        self.wall_held[slot] = (i, hs, hr, ht)
        nxf = -ap * _cross(n, ft)
        f.index_add_(0, i, fn + ft)
        t.index_add_(0, i, nxf - mr - mt if memory else nxf)
        return fn + ft, mr, mt

    def walls(self, p, arm, v, w, f, t):
        zero = torch.zeros(3, dtype=torch.float64, device=self.dev)
        if self.cube is not None:
            for a in range(3):
                e, h = p[:, a] - self.cube["centre"][a], self.cube["half"][a]
                for s in (1.0, -1.0):
                    i = torch.nonzero((s * e > 0) & (s * e + self.r[:, 0] - h > 0))[:, 0]
                    ap = (h - s * e[i])[:, None]
                    n = torch.zeros(len(i), 3, dtype=torch.float64, device=self.dev)
                    n[:, a] = -s
                    self.one_sided((a, s), i, n, ap, self.r[i] - ap, arm, v, w, f, t, zero, self.r[i], self.m[i], 2.0,
                                   self.memory)
        if self.cyl is not None:
            R, H = self.cyl["radius"], self.cyl["half_height"]
            e = p - torch.as_tensor(self.cyl["centre"], dtype=torch.float64, device=self.dev)
            flat = e.clone()
            flat[:, 2] = 0
            rho = flat.norm(dim=1)
            for s in (-1.0, 1.0):
                i = torch.nonzero((e[:, 2].abs() - H + self.r[:, 0] >= 1e-14) & (s * e[:, 2] > 0))[:, 0]
                ap = (H - s * e[i, 2])[:, None]
                n = torch.zeros(len(i), 3, dtype=torch.float64, device=self.dev)
                n[:, 2] = -s
                self.one_sided(("cap", s), i, n, ap, self.r[i] - ap, arm, v, w, f, t, zero, self.r[i], self.m[i], 2.0)
            i = torch.nonzero(rho - R + self.r[:, 0] >= 1e-14)[:, 0]
            ap = (R - rho[i])[:, None]
            self.one_sided("side", i, -flat[i] / rho[i, None], ap, self.r[i] - ap, arm, v, w, f, t, zero, self.r[i],
                           self.m[i], 2.0)

    def intruder(self, p, arm, v, w, f, t):
        R = self.intr["R"]
        d = p - self.intr["p"]
        dist = d.norm(dim=1)
        i = torch.nonzero(self.r[:, 0] - (dist - R) > 0)[:, 0]
        n, ap = d[i] / dist[i, None], (dist[i] - R)[:, None]
        ri = self.r[i]
        fi, mr, mt = self.one_sided("intruder", i, n, ap, ri - ap, arm, v, w, f, t, self.intr["v"], ri * R / (ri + R),
                                    self.m[i], 1.0)
        self.record.append(torch.cat([-fi.sum(0), (_cross(fi, R * n) + mr + mt).sum(0)]))

    def clumps(self):
        return {"pos": self.X, "vel": self.V, "angvel": self.W, "force": self.F, "torque": self.T, "quat": self.Q}


def _exact_run(scene, steps):
    e = _Exact(scene, "cuda" if torch.cuda.is_available() else "cpu")
    for _ in range(steps):
        e.step()
    return e


def exact(case, seed):
    if case["kind"] == "sort":
        return None
    if case["kind"] == "batch":
        got = [_exact_run(sc, case["steps"]).clumps() for sc in _uneven(case, seed)]
        out = {k: torch.cat([g[k] for g in got]).cpu().numpy() for k in got[0]}
        out["stats"] = None
        return out
    if case["kind"] == "serve":
        curve, pos = [], []
        for sc, n in zip(_uneven(case, seed), _request_steps(case)):
            e = _exact_run(sc, n)
            curve += [e.record[k - 1].cpu().numpy() for k in range(1, n + 1) if k % 50 == 0 or k == n]
            pos.append(e.intr["p"].cpu().numpy())
        return {"curve": np.array(curve), "pos": np.array(pos), "steps": None}
    e = _exact_run(_scene(case, seed), case["steps"])
    out = {k: v.cpu().numpy() for k, v in e.clumps().items()}
    out["stats"] = None
    if case.get("rows"):
        out["rows"] = out["front"] = out["back"] = None
    if case.get("intruder_mm"):
        out["curve"] = torch.stack(e.record).cpu().numpy()
    return out
