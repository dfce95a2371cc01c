"""Timed cases of the granular engine: whole jobs through the public front end.

A case is one job as a user's program runs it: create the engine from host
arrays (Engine / SqEngine), setup(), run(steps), and read the state back.  The
scenes are the framework's configurations (sphere pour, conical hopper,
rotating drum, large bed over a triangulated floor, a mixture of small and
large spheres, a superquadric packing) at sizes from the smallest jobs of the
tests to the bench's million-particle states, generated here from a seed.

Sphere scenes stand on a close-packed lattice of spacing a whose radii scatter
by +-0.1 % around a / 2 (with a share of smaller spheres where the
configuration is polydisperse), so about half of the near neighbours touch,
with the small overlaps of a bed at rest.

``exact`` computes the same job in plain torch, FP64, without the engine: the
half-list history rules, periodic images and walls are restated on the whole
pair list; triangulated walls are treated as the facets they approximate.
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.abspath(__file__)), "..", "liggghts-public_b200", "python"))
import granb200  # noqa: E402

PIN = ("x", "v", "omega", "radius", "rmass", "type", "tag")


def listed():
    return [
        # the smallest job: a test-size pour, where launches and latency are everything
        {"name": "pour_1500", "kind": "pour", "n": 1500, "steps": 400, "precision": "fp64", "rolling": False},
        # configuration 1: the 20,000-sphere pour in a periodic box
        {"name": "pour_20k", "kind": "pour", "n": 20000, "steps": 400, "precision": "fp64", "rolling": False},
        # a fast pour with rolling friction: ghosts, and a neighbour rebuild every ~50 steps
        {"name": "pour_300k_rolling", "kind": "pour", "n": 300001, "steps": 150, "precision": "fp64",
         "rolling": True},
        # a small mesh hopper, as users debug one
        {"name": "hopper_6k", "kind": "hopper", "n": 6000, "steps": 400, "precision": "fp64"},
        # configuration 2, the headline: 1M spheres, rolling friction, 8,192-triangle cone
        {"name": "hopper_1m", "kind": "hopper", "n": 1000000, "steps": 100, "precision": "fp64"},
        # the same in split precision
        {"name": "hopper_1m_split", "kind": "hopper", "n": 1000000, "steps": 100, "precision": "split"},
        # a bench-top drum: moving mesh, forced rebuilds
        {"name": "drum_40k", "kind": "drum", "n": 40009, "steps": 250, "precision": "fp64"},
        # configuration 3's drum at an eighth of its size, split precision
        {"name": "drum_1m_split", "kind": "drum", "n": 1000000, "steps": 100, "precision": "split"},
        # configuration 5's close-packed bed (12 contacts each) at a tenth of its size
        {"name": "bed_2m", "kind": "bed", "n": 2000000, "steps": 50, "precision": "fp64"},
        # strongly bidisperse bed: lists of more than 64 entries
        {"name": "mixture_8k", "kind": "mixture", "n": 8000, "steps": 300, "precision": "fp64"},
        # superquadrics: a small packing and configuration 4's 200,000
        {"name": "sq_2k", "kind": "sq", "n": 2000, "steps": 60, "precision": "fp64"},
        {"name": "sq_200k", "kind": "sq", "n": 200000, "steps": 20, "precision": "fp64"},
    ]


#: per kind: smallest and largest particle number, particle-steps of one pass at most
RANGES = {"pour": (1500, 300001, 4.5e7), "hopper": (6000, 1000000, 1e8), "drum": (6000, 1000000, 1e8),
          "bed": (20000, 2000000, 1e8), "mixture": (4000, 60000, 6e6), "sq": (300, 200000, 4e6)}


def draw(rng):
    kind = rng.choice(("pour", "pour", "hopper", "hopper", "drum", "bed", "mixture", "sq"))
    lo, hi, most = RANGES[kind]
    n = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    top = 60 if kind == "sq" else 400
    steps = max(10, min(top, int(most / n), rng.randint(top // 4, top)))
    case = {"kind": kind, "n": n, "steps": steps,
            "precision": "fp64" if kind in ("sq", "mixture") else rng.choice(("fp64", "fp64", "split"))}
    if kind == "pour":
        case["rolling"] = rng.random() < 0.5
    return case


# ---------------------------------------------------------------- scenes

def _sites(a, n, inside, lo, hi):
    """n sites of a hexagonal close packing of spacing a, from the bottom up, where inside(x, y, z) holds."""
    dy, dz = 0.5 * math.sqrt(3.0) * a, math.sqrt(2.0 / 3.0) * a
    nx, ny = int((hi[0] - lo[0]) / a) + 1, int((hi[1] - lo[1]) / dy) + 1
    i, j = np.meshgrid(np.arange(nx), np.arange(ny), indexing="xy")
    got, have, k = [], 0, 0
    while have < n:
        x = lo[0] + a * (i + 0.5 * ((j + k) % 2))
        y = lo[1] + dy * j + (k % 2) * dy / 3.0
        z = np.full(x.shape, lo[2] + k * dz)
        if z[0, 0] > hi[2]:
            raise ValueError("the packing does not fit")
        ok = inside(x, y, z) & (x <= hi[0]) & (y <= hi[1])
        p = np.stack([x[ok], y[ok], z[ok]], axis=1)
        got.append(p)
        have += len(p)
        k += 1
    return np.concatenate(got)[:n]


def _radii(rng, a, n, small):
    r = 0.5 * a * (1.0 + rng.uniform(-1e-3, 1e-3, n))
    pick = rng.random(n) < small
    r[pick] = rng.uniform(0.25 * a, 0.5 * a, int(pick.sum()))
    return r


def _scene(rng, dt, lo, hi, periodic, rolling, E, e, mu, density, x, v, r, fixes, skin=0.5e-3):
    n = len(r)
    atoms = {"x": x, "v": v, "omega": rng.uniform(-5.0, 5.0, (n, 3)), "radius": r,
             "rmass": 4.0 * math.pi / 3.0 * r * r * r * density,
             "type": np.ones(n, dtype=np.int32), "tag": np.arange(1, n + 1, dtype=np.int32)}
    one = np.ones((1, 1))
    return {"dt": dt, "skin": skin, "boxlo": [float(c) for c in lo], "boxhi": [float(c) for c in hi],
            "periodic": periodic, "every": 1, "delay": 0, "check": 1, "sortfreq": 1000, "sortbinsize": 0.0,
            "rolling_cdt": int(rolling), "tangential_damping": 1, "ntypes": 1, "youngs": np.array([E]),
            "poisson": np.array([0.45]), "restitution": e * one, "friction": mu * one, "rollfriction": 0.1 * one,
            "atoms": atoms, "fixes": [{"kind": "gravity", "magnitude": 9.81, "vector": [0.0, 0.0, -1.0]}] + fixes +
            [{"kind": "nve_sphere"}]}


def _pour(n, rng, rolling):
    s = 2.2e-3   # spheres of radius 1 mm a fifth of a radius apart, falling and colliding
    m = max(8, int(round((0.5 * n) ** (1.0 / 3.0))))
    i = np.arange(n)
    x = np.stack([(i % m + 0.5) * s, (i // m % m + 0.5) * s, 1.1e-3 + i // (m * m) * s], axis=1)
    x += rng.uniform(-0.08e-3, 0.08e-3, x.shape)
    v = rng.uniform(-0.3, 0.3, x.shape)
    v[:, 2] -= 0.2
    return _scene(rng, 1e-5, [0, 0, 0], [m * s, m * s, x[:, 2].max() + 0.02], [1, 1, 0], rolling, 5e6, 0.3, 0.5, 2500.0, x,
                  v, np.full(n, 1e-3), [{"kind": "wall_plane", "dim": 2, "pos": 0.0, "wall_type": 1,
                                         "rolling_cdt": int(rolling)}])


def _push(x, r, gap, direction, reach):
    """Spheres whose gap to the wall is below reach of their radius, moved onto it (overlap 0.1 % of the radius)."""
    near = gap < reach * r
    x[near] += ((gap[near] + 1e-3 * r[near]))[:, None] * direction[near]


def _quads(p):
    """Two triangles per cell of a grid of points (m, k, 3)."""
    a, b, c, d = p[:-1, :-1], p[:-1, 1:], p[1:, :-1], p[1:, 1:]
    t = np.stack([np.stack([a, b, d], axis=2), np.stack([a, d, c], axis=2)], axis=2)
    return np.ascontiguousarray(t.reshape(-1, 3, 3))


def _ring(n_theta):
    th = np.arange(n_theta + 1) % n_theta * (2.0 * math.pi / n_theta)
    return np.cos(th), np.sin(th)


def _hopper(n, rng):
    a, r_out, tan = 2e-3, 0.015, math.tan(math.radians(60.0))
    n_theta, n_z = (128, 32) if n >= 50000 else (48, 12)
    c = math.cos(math.pi / n_theta)
    height = ((n * a ** 3 / math.sqrt(2.0)) * 3.0 / (math.pi * tan * tan)) ** (1.0 / 3.0) + 6 * a
    rtop = r_out + height * tan

    def facet(x, y):
        k = np.floor(np.arctan2(y, x) / (2.0 * math.pi / n_theta))
        m = (k + 0.5) * (2.0 * math.pi / n_theta)
        return np.cos(m), np.sin(m)

    def dist(x, y, z):   # to the facet of the cone at this angle
        cx, cy = facet(x, y)
        return ((r_out + z * tan) * c - x * cx - y * cy) / math.sqrt(1.0 + (tan * c) ** 2)

    def inside(x, y, z):   # what has begun to fall out is clear of the outlet's rim
        free = np.where(z < 6e-3, np.hypot(x, y) <= r_out * c - 1.2e-3, True)
        return free & (dist(x, y, z) >= 0.5 * a * (1.0 + 2e-3))

    x = _sites(a, n, inside, [-rtop, -rtop, 0.5 * a], [rtop, rtop, height])
    r = _radii(rng, a, n, 0.25)
    cx, cy = facet(x[:, 0], x[:, 1])
    out = np.stack([cx, cy, np.full(n, -tan * c)], axis=1) / math.sqrt(1.0 + (tan * c) ** 2)
    _push(x, r, dist(x[:, 0], x[:, 1], x[:, 2]) - r, out, 0.15)
    v = rng.uniform(-0.02, 0.02, x.shape)
    v[:, 2] -= 0.6 * (r_out / (r_out + x[:, 2] * tan)) ** 2   # the discharge, fastest at the outlet
    cs, sn = _ring(n_theta)
    zs = np.linspace(0.0, height + 0.01, n_z + 1)
    rr = (r_out + zs * tan)[:, None]
    nodes = _quads(np.stack([rr * cs, rr * sn, np.broadcast_to(zs[:, None], (n_z + 1, n_theta + 1))], axis=2))
    w = rtop + 0.05
    return _scene(rng, 5e-6, [-w, -w, -0.09], [w, w, height + 0.03], [0, 0, 0], True, 5e6, 0.3, 0.5, 2500.0, x, v, r,
                  [{"kind": "wall_mesh", "nodes": nodes, "wall_type": 1, "curvature": 0.0, "rolling_cdt": 1,
                    "facets": "cone", "n_theta": n_theta, "r_out": r_out, "tan": tan},
                   {"kind": "wall_plane", "dim": 2, "pos": -0.08, "wall_type": 1, "rolling_cdt": 1}])


def _drum(n, rng):
    a, omega = 2e-3, 2.0
    R = (n * a ** 3 / math.sqrt(2.0) / (0.33 * math.pi * 3.4)) ** (1.0 / 3.0) + 2 * a
    L = 3.4 * R
    n_theta, n_ax, rings = (128, 121, 4) if n >= 200000 else (48, 12, 3)
    ap = R * math.cos(math.pi / n_theta)

    def facet(y, z):
        m = (np.floor(np.arctan2(z, y) / (2.0 * math.pi / n_theta)) + 0.5) * (2.0 * math.pi / n_theta)
        return np.cos(m), np.sin(m)

    def dist(y, z):
        cy, cz = facet(y, z)
        return ap - y * cy - z * cz

    x = _sites(a, n, lambda x, y, z: dist(y, z) >= 0.5 * a * (1.0 + 2e-3), [-0.5 * L + 0.51 * a, -R, -R], [0.5 * L - 0.51 * a, R, R])
    r = _radii(rng, a, n, 0.25)
    cy, cz = facet(x[:, 1], x[:, 2])
    _push(x, r, dist(x[:, 1], x[:, 2]) - r, np.stack([np.zeros(n), cy, cz], axis=1), 0.15)
    v = rng.uniform(-0.02, 0.02, x.shape)   # the bed turns with the drum
    v[:, 1] -= omega * x[:, 2]
    v[:, 2] += omega * x[:, 1]
    cs, sn = _ring(n_theta)
    xs = np.linspace(-0.5 * L, 0.5 * L, n_ax + 1)
    side = _quads(np.stack([np.broadcast_to(xs[:, None], (n_ax + 1, n_theta + 1)), np.broadcast_to(R * cs, (n_ax + 1, n_theta + 1)),
                            np.broadcast_to(R * sn, (n_ax + 1, n_theta + 1))], axis=2))
    caps = []
    for x0 in (-0.5 * L, 0.5 * L):
        rr = (np.arange(1, rings + 1) / rings * R)[:, None]
        caps.append(_quads(np.stack([np.full((rings, n_theta + 1), x0), rr * cs, rr * sn], axis=2)))
        p = np.stack([np.full(n_theta + 1, x0), R / rings * cs, R / rings * sn], axis=1)
        caps.append(np.stack([np.broadcast_to([x0, 0.0, 0.0], (n_theta, 3)), p[:-1], p[1:]], axis=1))
    nodes = np.ascontiguousarray(np.concatenate([side] + caps))
    lo, hi = [-0.5 * L - 0.01, -R - 0.01, -R - 0.01], [0.5 * L + 0.01, R + 0.01, R + 0.01]
    return _scene(rng, 5e-6, lo, hi, [0, 0, 0], False, 1e7, 0.5, 0.4, 2700.0, x, v, r,
                  [{"kind": "wall_mesh", "nodes": nodes, "wall_type": 1, "curvature": 0.0, "rolling_cdt": 0,
                    "facets": "drum", "n_theta": n_theta, "R": R, "L": L, "omega": omega},
                   {"kind": "move_mesh_rotate", "mesh": 1, "origin": [0.0, 0.0, 0.0], "axis": [1.0, 0.0, 0.0],
                    "period": 2.0 * math.pi / omega}])


def _bed(n, rng):
    a = 1e-3
    m = int(math.ceil((n / 1.2) ** (1.0 / 3.0)))
    side = m * a
    x = _sites(a, n, lambda x, y, z: (x <= side - 0.49 * a) & (y <= side - 0.49 * a), [0.5 * a, 0.5 * a, 0.5 * a], [side, side, 1e9])
    r = 0.5 * a * (1.0 + rng.uniform(0.0, 1e-3, n))   # every neighbour touches
    v = rng.uniform(-0.02, 0.02, x.shape)
    g = np.linspace(-2.13e-3, side + 2.29e-3, 129 if n >= 200000 else 33)
    gx, gy = np.meshgrid(g, g, indexing="ij")
    floor = _quads(np.stack([gx, gy, np.zeros_like(gx)], axis=2))
    walls = [{"kind": "wall_plane", "dim": d, "pos": p, "wall_type": 1} for d in (0, 1) for p in (0.0, side)]
    return _scene(rng, 2e-6, [-0.005] * 3, [side + 0.005, side + 0.005, x[:, 2].max() + 0.01], [0, 0, 0], False, 5e6, 0.3,
                  0.5, 2500.0, x, v, r, [{"kind": "wall_mesh", "nodes": floor, "wall_type": 1, "curvature": 0.0,
                                          "facets": "floor"}] + walls)


def _mixture(n, rng):
    s, rs, rb = 0.68e-3, 0.3e-3, 3e-3
    m = max(20, int(round((2.5 * n) ** (1.0 / 3.0))))
    i = np.arange(n + 2 * 800)
    x = np.stack([(i % m + 0.5) * s, (i // m % m + 0.5) * s, rs + 0.05e-3 + i // (m * m) * s], axis=1)
    x += rng.uniform(-0.04e-3, 0.04e-3, x.shape)
    L, zm = m * s, 0.5 * x[:, 2].max()
    big = np.array([[0.25 * L, 0.5 * L, zm], [0.75 * L, 0.5 * L, zm]])
    keep = np.ones(len(x), dtype=bool)
    for c in big:
        keep &= np.linalg.norm(x - c, axis=1) > rb + rs + 0.05e-3
    x = np.concatenate([big, x[keep]])[:n]
    r = np.concatenate([np.full(2, rb), np.full(len(x) - 2, rs)])
    return _scene(rng, 2e-6, [0, 0, 0], [L, L, x[:, 2].max() + 0.012], [1, 1, 0], True, 5e6, 0.3, 0.5, 2500.0, x,
                  rng.uniform(-0.3, 0.3, x.shape), r, [{"kind": "wall_plane", "dim": 2, "pos": 0.0, "wall_type": 1,
                                                       "rolling_cdt": 1}])


def _beta(p, q):
    p, q = torch.from_numpy(p), torch.from_numpy(q)
    return torch.exp(torch.lgamma(p) + torch.lgamma(q) - torch.lgamma(p + q)).numpy()


def _sq(n, rng):
    shape, blk = rng.uniform(1e-3, 2e-3, (n, 3)), rng.uniform(2.0, 8.0, n)
    q = rng.standard_normal((n, 4))
    q /= np.linalg.norm(q, axis=1)[:, None]
    m = int(math.ceil(n ** (1.0 / 3.0)))
    i = np.arange(n)
    x = np.stack([i % m, i // m % m, i // (m * m)], axis=1) * (1.42 * math.sqrt(12.0) * 1e-3)
    e = 2.0 / blk
    a, b, c = shape.T
    vol = 2.0 * a * b * c * e * e * _beta(0.5 * e, e + 1.0) * _beta(0.5 * e, 0.5 * e + 1.0)
    t1, t2 = _beta(1.5 * e, 0.5 * e) * _beta(0.5 * e, 2.0 * e + 1.0), 4.0 * _beta(0.5 * e, 0.5 * e + 1.0) * _beta(1.5 * e, e + 1.0)
    inertia = (1250.0 * a * b * c * e * e)[:, None] * np.stack([b * b * t1 + c * c * t2, a * a * t1 + c * c * t2,
                                                               (a * a + b * b) * t1], axis=1)
    return {"dt": 1e-5, "skin": 0.5e-3, "youngs": 5e6, "poisson": 0.45, "restitution": 0.3, "friction": 0.5,
            "atoms": {"x": x - x.mean(axis=0), "v": rng.uniform(-1.0, 1.0, (n, 3)), "quat": q, "angmom": np.zeros((n, 3)),
                      "shape": shape, "blockiness": blk, "rmass": vol * 2500.0, "inertia": inertia, "volume": vol}}


def scene(case, seed):
    rng = np.random.default_rng(seed)
    kind, n = case["kind"], case["n"]
    if kind == "pour":
        return _pour(n, rng, case["rolling"])
    return {"hopper": _hopper, "drum": _drum, "bed": _bed, "mixture": _mixture, "sq": _sq}[kind](n, rng)


# ---------------------------------------------------------------- the job

def prepare(case, seed):
    """The job's host arrays, the atoms in page-locked memory, and room for its result."""
    sc = scene(case, seed)
    if case["kind"] == "sq":
        return {"case": case, "scene": sc}
    for k in PIN:
        p = granb200.pinned_empty(sc["atoms"][k].shape, sc["atoms"][k].dtype)
        p[...] = sc["atoms"][k]
        sc["atoms"][k] = p
    n = len(sc["atoms"]["tag"])
    out = {k: granb200.pinned_empty((n, 3)) for k in ("x", "v", "omega", "f", "torque")}
    out["tag"] = granb200.pinned_empty((n,), np.int32)
    return {"case": case, "scene": sc, "out": out}


def run(state):
    case, sc = state["case"], state["scene"]
    if case["kind"] == "sq":
        eng = granb200.SqEngine(sc)
    else:
        eng = granb200.Engine(sc, precision=granb200.PREC_SPLIT if case["precision"] == "split" else granb200.PREC_FP64)
    eng.setup()
    eng.run(case["steps"])
    res = eng.atoms() if case["kind"] == "sq" else eng.atoms(state["out"])
    eng.close()
    return res


#: touching pairs a particle (both sides counted once), wall contacts a particle
PAIRS = {"pour": 0.3, "hopper": 2.0, "drum": 2.0, "bed": 5.8, "mixture": 0.3, "sq": 0.15}


def work(case):
    """Bytes: the state in and out over the bus, and every step its own records once (position, velocity, angular
    velocity, mass, type and the neighbour indices read, the moved ones written, the shear history of the touching
    pairs read and written).  Flops: ~250 per touching pair, ~60 per particle and step."""
    n, steps, pairs = case["n"], case["steps"], PAIRS[case["kind"]] * case["n"]
    if case["kind"] == "sq":   # a Newton solve of ~5 iterations of ~600 operations per contact
        return {"bytes": n * (200 + 184) + steps * (n * 400 + pairs * 200), "flops": steps * (pairs * 3000 + n * 300)}
    return {"bytes": n * (96 + 124) + steps * (n * (92 + 72 + 24 + 24) + pairs * 52), "flops": steps * (pairs * 250 + n * 60)}


def tolerance(case):
    """FP64 spheres repeat the reference's arithmetic bit for bit.  Split precision: FP32 contact sums (a pair on the
    Coulomb cap can take the other branch), 1e-3 from FP64 at most over these jobs.  Superquadrics: a solve ends at
    merit 1e-10, an angle of 1e-5, and the jobs end 2.5e-3 at most from converged solves."""
    if case["kind"] == "sq":
        return {"rel": 1e-2, "max": 0.9}
    if case["precision"] == "split":
        return {"rel": 4e-3, "max": 0.9}
    return "exact"


# ---------------------------------------------------------------- the same job in plain torch, FP64

DEV = "cuda" if torch.cuda.is_available() else "cpu"


def _t(a):
    return torch.from_numpy(np.array(a)).to(DEV)


def _cell_pairs(x, reach, cut, box, periodic, lo):
    """Pairs i < j whose minimum-image distance is below reach(i, j)."""
    n = len(x)
    nc = [max(1, min(1024, int(box[d] / cut))) for d in range(3)]
    c = [torch.clamp(((x[:, d] - lo[d]) / box[d] * nc[d]).long(), 0, nc[d] - 1) for d in range(3)]
    key = (c[2] * nc[1] + c[1]) * nc[0] + c[0]
    order = torch.argsort(key)
    cnt = torch.bincount(key, minlength=nc[0] * nc[1] * nc[2])
    start = torch.cumsum(cnt, 0) - cnt
    me, pi, pj = torch.arange(n, device=x.device), [], []
    offs = [sorted({o if nc[d] > 2 or not periodic[d] else o % nc[d] for o in (-1, 0, 1)}) for d in range(3)]
    for oz in offs[2]:
        for oy in offs[1]:
            for ox in offs[0]:
                ok = torch.ones(n, dtype=torch.bool, device=x.device)
                cc = []
                for d, o in ((0, ox), (1, oy), (2, oz)):
                    k = c[d] + o
                    if periodic[d]:
                        k = k % nc[d]
                    else:
                        ok &= (k >= 0) & (k < nc[d])
                    cc.append(torch.clamp(k, 0, nc[d] - 1))
                other = (cc[2] * nc[1] + cc[1]) * nc[0] + cc[0]
                left = torch.where(ok, cnt[other], torch.zeros_like(other))
                for s in range(int(left.max())):
                    i = me[left > s]
                    j = order[start[other[i]] + s]
                    i, j = i[j > i], j[j > i]
                    d = _image(x[i] - x[j], box, periodic)
                    near = (d * d).sum(1) < reach(i, j) ** 2
                    pi.append(i[near])
                    pj.append(j[near])
    return torch.cat(pi), torch.cat(pj)


def _image(d, box, periodic):
    for k in range(3):
        if periodic[k]:
            d[:, k] -= box[k] * torch.round(d[:, k] / box[k])
    return d


def _contact(M, d, r, delta, en, reff, meff, vrel, cw, roll, sh, upd, dt):
    """Hertz normal force, history tangential force, CDT rolling torque: force, friction torque direction, roll."""
    vn = (vrel * en).sum(1, keepdim=True)
    vt = vrel - vn * en + torch.linalg.cross(d, cw)
    root = torch.sqrt(reff * delta)
    kn, kt = 4.0 / 3.0 * M["Y"] * root, 8.0 * M["G"] * root
    c = -2.0 * math.sqrt(5.0 / 6.0) * M["beta"]
    fn = -c * torch.sqrt(2.0 * M["Y"] * root * meff) * vn[:, 0] + kn * delta
    if upd:
        sh = sh + vt * dt
        sh = sh - (sh * en).sum(1, keepdim=True) * en
    mag = torch.linalg.norm(sh, dim=1)
    ft = -kt[:, None] * sh
    cap = M["mu"] * fn.abs()
    slip = kt * mag > cap
    lim = ft * (cap / torch.clamp(kt * mag, min=1e-300))[:, None]
    if upd:
        sh = torch.where(slip[:, None], -lim / kt[:, None], sh)
    ft = torch.where(slip[:, None], lim, ft - (c * torch.sqrt(kt * meff))[:, None] * vt)
    rt = torch.zeros_like(ft)
    if roll is not None:
        wm = torch.linalg.norm(roll, dim=1)
        rt = torch.where((wm > 0)[:, None], (M["mur"] * kn * delta * reff / torch.clamp(wm, min=1e-300))[:, None] * roll,
                         rt)
        rt = rt - (rt * en).sum(1, keepdim=True) * en
    return fn[:, None] * en + ft, torch.linalg.cross(en, ft), rt, sh


def _facets(f, x, r, t):
    """(wall key, distance of the centre to the wall, direction from the wall to the centre) of a triangulated wall."""
    if f["facets"] == "floor":
        yield 0, x[:, 2], torch.tensor([0.0, 0.0, 1.0], dtype=x.dtype, device=x.device).expand_as(x)
        return
    w = 2.0 * math.pi / f["n_theta"]
    drum = f["facets"] == "drum"
    turn = f["omega"] * t if drum else 0.0
    a, b = (x[:, 1], x[:, 2]) if drum else (x[:, 0], x[:, 1])
    k0 = torch.floor((torch.atan2(b, a) - turn) / w)
    for o in range(-3, 4):   # near the outlet a sphere is wider than a facet
        m, sgn = (k0 + o + 0.5) * w + turn, (o > 0) - (o < 0)
        cx, cy = torch.cos(m), torch.sin(m)
        along, side = a * cx + b * cy, b * cx - a * cy   # in the facet's frame
        c = math.cos(math.pi / f["n_theta"])
        if drum:
            dist, en, at = f["R"] * c - along, torch.stack([torch.zeros_like(cx), -cx, -cy], 1), f["R"] * c
        else:
            s = math.sqrt(1.0 + (f["tan"] * c) ** 2)
            dist = ((f["r_out"] + x[:, 2] * f["tan"]) * c - along) / s
            en = torch.stack([-cx, -cy, torch.full_like(cx, f["tan"] * c)], 1) / s
            at = along + dist / s
        inside = side.abs() <= at * math.tan(math.pi / f["n_theta"])
        # beyond the facet: its edge towards the sphere, which of the two facets there the one of larger index owns
        me, him = torch.remainder(k0 + o - sgn, f["n_theta"]), torch.remainder(k0 + o, f["n_theta"])
        ex, ey = torch.cos(m - 0.5 * sgn * w), torch.sin(m - 0.5 * sgn * w)
        if drum:
            away = torch.stack([torch.zeros_like(ex), a - f["R"] * ex, b - f["R"] * ey], 1)
        else:
            u = torch.stack([f["tan"] * ex, f["tan"] * ey, torch.ones_like(ex)], 1) / math.sqrt(1.0 + f["tan"] ** 2)
            away = x - torch.stack([f["r_out"] * ex, f["r_out"] * ey, torch.zeros_like(ex)], 1)
            away = away - (away * u).sum(1, keepdim=True) * u
        edge = torch.linalg.norm(away, dim=1)
        edge = torch.where(him > me, edge, torch.full_like(edge, 1e9))
        dist, en = torch.where(inside, dist, edge), torch.where(inside[:, None], en, away / edge[:, None])
        if not drum:   # below the outlet: its rim
            foot = x - dist[:, None] * en
            rim = torch.stack([f["r_out"] * c * cx - side * cy, f["r_out"] * c * cy + side * cx, torch.zeros_like(cx)], 1)
            rim = torch.where(inside[:, None], rim, f["r_out"] * torch.stack([ex, ey, torch.zeros_like(ex)], 1))
            away = x - rim
            far = torch.linalg.norm(away, dim=1)
            low = (foot[:, 2] < 0) & (dist < 1e8)
            dist, en = torch.where(low, far, dist), torch.where(low[:, None], away / far[:, None], en)
        yield o, dist, en
    if drum:
        for key, sgn in ((8, 1.0), (9, -1.0)):
            en = torch.tensor([sgn, 0.0, 0.0], dtype=x.dtype, device=x.device).expand_as(x)
            yield key, 0.5 * f["L"] + sgn * x[:, 0], en


def _walls(sc, M, x, v, w, r, m, hist, upd, t, F, T):
    for q, f in enumerate(sc["fixes"]):
        if f["kind"] == "wall_plane":
            d = x[:, f["dim"]] - f["pos"]
            en = torch.zeros_like(x)
            en[:, f["dim"]] = torch.sign(d)
            items = [(0, d.abs(), en)]
        elif f["kind"] == "wall_mesh":
            items = _facets(f, x, r, t)
        else:
            continue
        for key, dist, en in items:
            i = torch.nonzero(dist <= r)[:, 0]
            old = hist.get((q, key))
            new = torch.zeros_like(x) if old is None or len(i) < len(x) else old
            if len(i):
                sh = new[i] if old is None else old[i]
                vw = torch.zeros((len(i), 3), dtype=x.dtype, device=x.device)
                if upd and f.get("facets") == "drum":   # the nodes have no velocity before the first step
                    p = x[i] - dist[i, None] * en[i]
                    vw[:, 1], vw[:, 2] = -f["omega"] * p[:, 2], f["omega"] * p[:, 1]
                e, over = en[i], r[i] - dist[i]
                cr = r[i] - 0.5 * over
                wr = cr[:, None] * w[i] / dist[i, None]
                Fi, tor, rt, sh = _contact(M, dist[i, None] * e, None, over, e, r[i], m[i], v[i] - vw, wr,
                                           wr if f.get("rolling_cdt") else None, sh, upd, sc["dt"])
                F[i] += Fi
                T[i] -= cr[:, None] * tor + rt
                if upd:
                    new[i] = sh
            if upd:
                hist[(q, key)] = new


def _exact_spheres(case, sc):
    at = {k: _t(sc["atoms"][k]) for k in ("x", "v", "omega", "radius", "rmass")}
    x, v, w, r, m = (at[k].clone() for k in ("x", "v", "omega", "radius", "rmass"))
    n, dt, skin = len(r), sc["dt"], sc["skin"]
    lo, hi = np.array(sc["boxlo"]), np.array(sc["boxhi"])
    box, per = hi - lo, sc["periodic"]
    E, nu, e = sc["youngs"][0], sc["poisson"][0], math.log(sc["restitution"][0, 0])
    M = {"Y": E / (2.0 * (1.0 - nu * nu)), "G": E / (4.0 * (2.0 - nu) * (1.0 + nu)), "beta": e / math.sqrt(e * e + math.pi ** 2),
         "mu": sc["friction"][0, 0], "mur": sc["rollfriction"][0, 0]}
    cutmax = 2.0 * float(r.max()) + skin
    # the order in which the engine keeps its atoms: stable by sort bin (half the neighbour cutoff), x fastest
    nb = [max(1, int(box[d] * (1.0 / (0.5 * cutmax)))) for d in range(3)]
    b = [np.clip(((sc["atoms"]["x"][:, d] - lo[d]) * (nb[d] / box[d])).astype(np.int64), 0, nb[d] - 1) for d in range(3)]
    order = torch.from_numpy(np.argsort((b[2] * nb[1] + b[1]) * nb[0] + b[0], kind="stable")).to(DEV)
    g = torch.tensor([0.0, 0.0, -9.81], dtype=x.dtype, device=DEV)
    pair = {"i": None}
    hist = {}

    def build():
        for d in range(3):
            if per[d]:
                x[:, d] = lo[d] + torch.remainder(x[:, d] - lo[d], box[d])
        i, j = _cell_pairs(x, lambda i, j: r[i] + r[j] + skin, cutmax, box, per, lo)
        key, by = torch.sort(i * n + j)
        i, j = i[by], j[by]
        sh = torch.zeros((len(i), 3), dtype=x.dtype, device=DEV)
        if pair["i"] is not None and len(pair["i"]):   # the history of pairs that touch at the rebuild
            d = _image(x[i] - x[j], box, per)
            touch = (d * d).sum(1) < (r[i] + r[j]) ** 2
            p = torch.clamp(torch.searchsorted(pair["key"], key), max=len(pair["key"]) - 1)
            sh = torch.where((touch & (pair["key"][p] == key))[:, None], pair["sh"][p], sh)
        pair.update(i=i, j=j, key=key, sh=sh, hold=x.clone())

    def force(upd, t):
        F, T = m[:, None] * g, torch.zeros_like(x)
        d = _image(x[pair["i"]] - x[pair["j"]], box, per)
        dist = torch.sqrt((d * d).sum(1))
        s = torch.nonzero(dist < r[pair["i"]] + r[pair["j"]])[:, 0]
        i, j, d, dist = pair["i"][s], pair["j"][s], d[s], dist[s]
        over = r[i] + r[j] - dist
        ci, cj = (r[i] - 0.5 * over)[:, None], (r[j] - 0.5 * over)[:, None]
        en = d / dist[:, None]
        Fi, tor, rt, sh = _contact(M, d, None, over, en, r[i] * r[j] / (r[i] + r[j]), m[i] * m[j] / (m[i] + m[j]),
                                   v[i] - v[j], (ci * w[i] + cj * w[j]) / dist[:, None],
                                   w[i] - w[j] if sc["rolling_cdt"] else None, pair["sh"][s], upd, dt)
        if upd:
            pair["sh"][s] = sh
        F.index_add_(0, i, Fi)
        F.index_add_(0, j, -Fi)
        T.index_add_(0, i, -ci * tor - rt)
        T.index_add_(0, j, -cj * tor + rt)
        _walls(sc, M, x, v, w, r, m, hist, upd, t, F, T)
        return F, T

    build()
    F, T = force(False, 0.0)
    half, rot = (0.5 * dt / m)[:, None], (0.5 * dt / 0.4 / (r * r * m))[:, None]
    for k in range(case["steps"]):
        v += half * F
        w += rot * T
        x += dt * v
        d = x - pair["hold"]
        if float((d * d).sum(1).max()) > 0.25 * skin * skin:
            build()
        F, T = force(True, (k + 1) * dt)
        v += half * F
        w += rot * T
    tag = (order + 1).to(torch.int32)
    out = {"x": x[order], "v": v[order], "omega": w[order], "f": F[order], "torque": T[order]}
    return {**{k: a.cpu().numpy() for k, a in out.items()}, "tag": tag.cpu().numpy()}


def _rot(q):
    w, i, j, k = q.unbind(1)
    return torch.stack([w * w + i * i - j * j - k * k, 2 * (i * j - k * w), 2 * (j * w + i * k), 2 * (i * j + k * w),
                        w * w - i * i + j * j - k * k, 2 * (j * k - i * w), 2 * (i * k - j * w), 2 * (j * k + i * w),
                        w * w - i * i - j * j + k * k], 1).view(-1, 3, 3)


def _mv(R, a):
    return (R @ a[:, :, None])[:, :, 0]


def _shape(body, p):
    """Superquadric shape function (scaled by 0.5^(n-2)), gradient and Hessian at p."""
    c, R, s, n = body
    u = _mv(R.transpose(1, 2), p - c) / s
    k, e = (0.5 ** (n - 2.0))[:, None], n[:, None]
    p2 = u.abs() ** (e - 2.0)
    f = k[:, 0] * ((p2 * u * u).sum(1) - 1.0)
    return f, _mv(R, k * e * p2 * u / s), R @ ((k * e * (e - 1.0) * p2 / (s * s))[:, :, None] * R.transpose(1, 2))


def _residual(A, B, p, mu):
    fa, ga, ha = _shape(A, p)
    fb, gb, hb = _shape(B, p)
    if mu is None:
        mu = torch.sqrt(((ga * gb).sum(1) / (gb * gb).sum(1)).abs())
    F = torch.cat([ga + (mu * mu)[:, None] * gb, (fa - fb)[:, None]], 1)
    return F, mu, (fa, fb, ga, gb, ha, hb)


def _pick(body, k):
    return tuple(b[k] for b in body)


def _newton(A, B, p, iters=60):
    """Contact points (gradients opposed, equal shape functions) of a batch of pairs, from the starts p."""
    F, mu, info = _residual(A, B, p, None)
    live = torch.arange(len(p), device=p.device)
    for _ in range(iters):
        if not len(live):
            break
        a, b, q, m = _pick(A, live), _pick(B, live), p[live], mu[live]
        F, _, (fa, fb, ga, gb, ha, hb) = _residual(a, b, q, m)
        J = torch.zeros((len(live), 4, 4), dtype=p.dtype, device=p.device)
        J[:, :3, :3] = ha + (m * m)[:, None, None] * hb
        J[:, :3, 3] = 2.0 * m[:, None] * gb
        J[:, 3, :3] = ga - gb
        step, bad = torch.linalg.solve_ex(J, F)
        step = torch.where((bad != 0)[:, None] | ~torch.isfinite(step), torch.zeros_like(step), step)
        size, now, on = torch.ones_like(m), (F * F).sum(1), torch.ones_like(m, dtype=torch.bool)
        best, bm = q.clone(), m.clone()
        for _ in range(12):   # halved until the residual falls
            t, tm = q - size[:, None] * step[:, :3], m - size * step[:, 3]
            Ft = _residual(a, b, t, tm)[0]
            ok = on & ((Ft * Ft).sum(1) < now)
            best[ok], bm[ok] = t[ok], tm[ok]
            on = on & ~ok
            size = size * 0.5
            if not bool(on.any()):
                break
        p[live], mu[live] = best, bm
        live = live[(~on) & (step[:, :3].abs().max(1).values > 1e-13 * a[2].min(1).values)]
    F, _, info = _residual(A, B, p, mu)
    return p, info, torch.linalg.cross(info[2], info[3]).pow(2).sum(1) / (info[2].pow(2).sum(1) * info[3].pow(2).sum(1))


def _contact_points(A, B, warm, start):
    """First contacts by the homotopy from spheres of equal volume scale, the others from their advanced point."""
    p = torch.zeros_like(A[0])
    k = torch.nonzero(warm)[:, 0]
    p[k] = _newton(_pick(A, k), _pick(B, k), start[k])[0]
    k = torch.nonzero(~warm)[:, 0]
    a, b = _pick(A, k), _pick(B, k)
    ra, rb = a[2].prod(1) ** (1.0 / 3.0), b[2].prod(1) ** (1.0 / 3.0)
    q = a[0] + (ra / (ra + rb))[:, None] * (b[0] - a[0])
    for i in range(11):
        t = i / 10.0
        at = lambda o, r: (o[0], o[1], r[:, None] + (o[2] - r[:, None]) * t, 2.0 + (o[3] - 2.0) * t)  # noqa: E731
        q = _newton(at(a, ra), at(b, rb), q)[0]
    p[k] = q
    return p


def _to_surface(body, p, d):
    """alpha with p + alpha d on the surface, p inside: bisection, then it is as exact as the numbers are."""
    lo, hi = torch.zeros(len(p), dtype=p.dtype, device=p.device), 2.0 * body[2].max(1).values
    for _ in range(70):
        mid = 0.5 * (lo + hi)
        inside = _shape(body, p + mid[:, None] * d)[0] < 0
        lo, hi = torch.where(inside, mid, lo), torch.where(inside, hi, mid)
    return 0.5 * (lo + hi)


def _quatvec(a, b):
    return torch.stack([-(a[:, 1:] * b).sum(1), a[:, 0] * b[:, 0] + a[:, 2] * b[:, 2] - a[:, 3] * b[:, 1],
                        a[:, 0] * b[:, 1] + a[:, 3] * b[:, 0] - a[:, 1] * b[:, 2],
                        a[:, 0] * b[:, 2] + a[:, 1] * b[:, 1] - a[:, 2] * b[:, 0]], 1)


def _body_momentum(q, p):
    """Body-frame angular momentum of the conjugate quaternion momentum p (the inverse of 2 q (x) L)."""
    return 0.5 * torch.stack([-q[:, 1] * p[:, 0] + q[:, 0] * p[:, 1] + q[:, 3] * p[:, 2] - q[:, 2] * p[:, 3],
                              -q[:, 2] * p[:, 0] - q[:, 3] * p[:, 1] + q[:, 0] * p[:, 2] + q[:, 1] * p[:, 3],
                              -q[:, 3] * p[:, 0] + q[:, 2] * p[:, 1] - q[:, 1] * p[:, 2] + q[:, 0] * p[:, 3]], 1)


def _turn(k, p, q, inertia, dt):
    sign, to = {1: ((-1, 1, 1, -1), (1, 0, 3, 2)), 2: ((-1, -1, 1, 1), (2, 3, 0, 1)),
                3: ((-1, 1, -1, 1), (3, 2, 1, 0))}[k]
    sg = torch.tensor(sign, dtype=p.dtype, device=p.device)
    kp, kq = sg * p[:, to], sg * q[:, to]
    phi = dt * (p * kq).sum(1, keepdim=True) / (4.0 * inertia[:, k - 1:k])
    c, s = torch.cos(phi), torch.sin(phi)
    return c * p + s * kp, c * q + s * kq


def _exact_sq(case, sc):
    at = {k: _t(a) for k, a in sc["atoms"].items()}
    x, v, q, L, s, n = (at[k].clone() for k in ("x", "v", "quat", "angmom", "shape", "blockiness"))
    m, inertia, dt, skin = at["rmass"], at["inertia"], sc["dt"], sc["skin"]
    rv = (0.75 * at["volume"] / math.pi) ** (1.0 / 3.0)
    E, nu, e = sc["youngs"], sc["poisson"], math.log(sc["restitution"])
    M = {"Y": E / (2.0 * (1.0 - nu * nu)), "G": E / (4.0 * (2.0 - nu) * (1.0 + nu)),
         "beta": e / math.sqrt(e * e + math.pi ** 2), "mu": sc["friction"]}
    rb = torch.linalg.norm(s, dim=1)
    cut, num = 2.0 * float(rb.max()) + skin, len(m)
    pair = {"key": None}

    def omega(R):
        return _mv(R, _mv(R.transpose(1, 2), L) / inertia)

    def build():
        lo = x.min(0).values.cpu().numpy() - 1e-6
        i, j = _cell_pairs(x, lambda i, j: rb[i] + rb[j] + skin, cut, x.max(0).values.cpu().numpy() + 1e-6 - lo,
                           [0, 0, 0], lo)
        key, by = torch.sort(i * num + j)
        i, j = i[by], j[by]
        sh, cp, touch = torch.zeros_like(x[i]), torch.zeros_like(x[i]), torch.zeros(len(i), dtype=torch.bool, device=DEV)
        if pair["key"] is not None and len(pair["key"]):
            p = torch.clamp(torch.searchsorted(pair["key"], key), max=len(pair["key"]) - 1)
            touch = (pair["key"][p] == key) & pair["touch"][p]
            sh, cp = torch.where(touch[:, None], pair["sh"][p], sh), pair["cp"][p]
        pair.update(i=i, j=j, key=key, sh=sh, cp=cp, touch=touch, hold=x.clone())

    def force(upd, w):
        F, T = torch.zeros_like(x), torch.zeros_like(x)
        d = x[pair["i"]] - x[pair["j"]]
        k = torch.nonzero((d * d).sum(1) < (rb[pair["i"]] + rb[pair["j"]]) ** 2)[:, 0]
        i, j, warm, old = pair["i"][k], pair["j"][k], pair["touch"][k], pair["cp"][k]
        R = _rot(q)
        A, B = (x[i], R[i], s[i], n[i]), (x[j], R[j], s[j], n[j])
        va = v[i] + torch.linalg.cross(w[i], old - x[i])
        vb = v[j] + torch.linalg.cross(w[j], old - x[j])
        p = _contact_points(A, B, warm, old + (va * m[i, None] + vb * m[j, None]) / (m[i] + m[j])[:, None] * dt)
        fa, ga, _ = _shape(A, p)
        fb, gb, _ = _shape(B, p)
        hit = torch.maximum(fa, fb) < 0
        pair["touch"][k], pair["cp"][k] = hit, p
        h = torch.nonzero(hit)[:, 0]
        k, i, j, p = k[h], i[h], j[h], p[h]
        en = gb[h] - ga[h]
        en = en / torch.linalg.norm(en, dim=1, keepdim=True)
        over = _to_surface(_pick(A, h), p, -en) + _to_surface(_pick(B, h), p, en)
        ai, aj = p - x[i], p - x[j]
        vrel = v[i] - v[j] + torch.linalg.cross(w[i], ai) - torch.linalg.cross(w[j], aj)
        Fi, _, _, sh = _contact(M, torch.zeros_like(en), None, over, en, rv[i] * rv[j] / (rv[i] + rv[j]),
                                m[i] * m[j] / (m[i] + m[j]), vrel, torch.zeros_like(en), None, pair["sh"][k], upd, dt)
        if upd:
            pair["sh"][k] = sh
        F.index_add_(0, i, Fi)
        F.index_add_(0, j, -Fi)
        T.index_add_(0, i, torch.linalg.cross(ai, Fi))
        T.index_add_(0, j, -torch.linalg.cross(aj, Fi))
        return F, T

    build()
    F, T = force(False, omega(_rot(q)))
    half = (0.5 * dt / m)[:, None]
    for _ in range(case["steps"]):
        v += half * F
        x += dt * v
        Rt = _rot(q).transpose(1, 2)
        p = 2.0 * _quatvec(q, _mv(Rt, L)) + dt * _quatvec(q, _mv(Rt, T))
        for k, h in ((3, 0.5), (2, 0.5), (1, 1.0), (2, 0.5), (3, 0.5)):
            p, q = _turn(k, p, q, inertia, h * dt)
        q = q / torch.linalg.norm(q, dim=1, keepdim=True)
        R = _rot(q)
        L = _mv(R, _body_momentum(q, p))
        d = x - pair["hold"]
        if float((d * d).sum(1).max()) > 0.25 * skin * skin:
            build()
        F, T = force(True, omega(R))
        v += half * F
        Rt = R.transpose(1, 2)
        L = _mv(R, _body_momentum(q, 2.0 * _quatvec(q, _mv(Rt, L)) + dt * _quatvec(q, _mv(Rt, T))))
    out = {"x": x, "v": v, "angmom": L, "omega": omega(_rot(q)), "f": F, "torque": T, "quat": q}
    return {k: a.cpu().numpy() for k, a in out.items()}


def exact(case, seed):
    sc = scene(case, seed)
    return _exact_sq(case, sc) if case["kind"] == "sq" else _exact_spheres(case, sc)
