"""Growth of the meshes' contact slots (32 triangles an atom at first, 64 at
most) while contacts exist: spheres slide along a floor whose triangles get
finer, and past a coarse upright wall (a second mesh), so that at some rebuild
an atom first has more than 32 candidate triangles while it touches the one
listed last.  Bit for bit against the oracle: during a run, at a restart, and
with the floor as the first or the second of two meshes."""
import os
import sys

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
for sub in ("../liggghts-public_b200/python", "../oracle"):
    p = os.path.join(HERE, sub)
    if p not in sys.path:
        sys.path.insert(0, p)
import gb2_scenarios as S  # noqa: E402
import oracle  # noqa: E402
from parity_util import assert_atoms_equal, assert_mesh_equal, assert_pairs_equal, mesh_contact_map  # noqa: E402

R, SKIN = 1e-3, 0.5e-3


def _strip(xs, ys, focus, upright=False):
    """Two triangles per cell of the grid xs x ys: on z = 0 facing up, or, upright, on y = 0 facing +y with
    ys along z.  The middle row of cells comes last, in each row the cells next to x = focus."""
    tris, rows = [], len(ys) - 1
    for b in sorted(range(rows), key=lambda b: -abs(2 * b - (rows - 1))):
        for a in sorted(range(len(xs) - 1), key=lambda a: -abs(0.5 * (xs[a] + xs[a + 1]) - focus)):
            p = [(xs[a], ys[b]), (xs[a + 1], ys[b]), (xs[a + 1], ys[b + 1]), (xs[a], ys[b + 1])]
            q = [(x, 0.0, y) if upright else (x, y, 0.0) for x, y in p]
            for t in ((0, 1, 2), (0, 2, 3)):
                tris.append([q[k] for k in (t[::-1] if upright else t)])
    return np.asarray(tris, dtype=np.float64)


def _scene(n=12, walls="floor"):
    """Spheres in a row along x, sliding at 1 m/s over the floor from cells of 1 x 0.9 mm to cells of 0.37 x 0.9 mm."""
    rng = np.random.default_rng(n)
    coarse = np.arange(-0.04, 0.0, 1e-3)
    xs = np.concatenate([coarse, np.arange(coarse[-1] + 0.37e-3, 0.02, 0.37e-3)])
    ys = R + (np.arange(6) - 2.5) * 0.9e-3
    pos = np.stack([-0.003 - 2.05 * R * np.arange(n), np.full(n, R - 1e-6), np.full(n, R - 2e-6)], axis=1)
    pos[:, 0] += rng.uniform(-1e-5, 1e-5, n)
    vel = np.zeros((n, 3))
    vel[:, 0] = 1.0 + rng.uniform(-0.01, 0.01, n)
    vel[:, 1] = -1e-3
    focus = coarse[-1] - R   # where the first sphere is when its list first outgrows 32
    floor = {"kind": "wall_mesh", "nodes": _strip(xs, ys, focus), "wall_type": 1, "curvature": 0.0}
    upright = {"kind": "wall_mesh", "nodes": _strip(np.arange(-0.04, 0.02, 0.9e-3), np.arange(-2e-3, 4.1e-3, 2e-3), focus, True),
               "wall_type": 1, "curvature": 0.0}
    meshes = {"floor": [floor], "floor_first": [floor, upright], "floor_last": [upright, floor]}[walls]
    sc = S.hopper(n=8, n_theta=12, n_z=4, seed=1)
    sc.update(name="mesh_slots", dt=2e-6, skin=SKIN, boxlo=[-0.05, -0.02, -0.02], boxhi=[0.05, 0.02, 0.02],
              periodic=[0, 0, 0], every=1, delay=0, check=1, sortfreq=0, rolling_cdt=0,
              atoms=S._atoms(pos, np.full(n, R), 2500.0, vel),
              fixes=[{"kind": "gravity", "magnitude": 9.81, "vector": [0.0, -0.3, -1.0]}] + meshes +
                    [{"kind": "nve_sphere"}])
    return sc


def _meshes(sc):
    return [k for k, f in enumerate(sc["fixes"]) if f["kind"] == "wall_mesh"]


def _close(nodes, x):
    """The triangles that a sphere at x lists (no further than R + SKIN / 2 off their plane and beyond each of
    their edges, TriMesh::resolveTriSphereNeighbuild), in order: their count, and the rank of the one below it."""
    c = nodes.mean(axis=1)
    n = np.cross(nodes[:, 1] - nodes[:, 0], nodes[:, 2] - nodes[:, 0])
    n /= np.linalg.norm(n, axis=1)[:, None]
    far = R + 0.5 * SKIN
    ok = np.abs(((x - c) * n).sum(axis=1)) <= far
    over = np.full(len(nodes), -np.inf)
    for k in range(3):
        e = np.cross(nodes[:, (k + 1) % 3] - nodes[:, k], n)
        d = ((x - nodes[:, k]) * e).sum(axis=1) / np.linalg.norm(e, axis=1)
        ok &= d <= far
        over = np.maximum(over, d)
    near = np.flatnonzero(ok)
    return len(near), int(np.argmin(over[near])) if len(near) else -1


def _check(e, o, sc):
    assert_atoms_equal(e, o)
    assert_pairs_equal(e, o)
    return [assert_mesh_equal(e, o, k) for k in _meshes(sc)]


def test_scene_reaches_the_growth():
    """What the GPU tests rest on, by the oracle and geometry alone: at the start no sphere lists more than 32
    triangles of any mesh; the first that does touches one beyond the 32nd, and so does some sphere at the end."""
    sc = _scene(walls="floor_last")
    o = oracle.Oracle(sc)
    o.setup()
    up, fl = (sc["fixes"][k]["nodes"] for k in _meshes(sc))
    assert max(_close(n, x)[0] for n in (up, fl) for x in o.atoms()["x"]) <= 32
    assert len(o.mesh_contacts(2)["tag"]) > 0
    first = None
    for _ in range(60):
        o.run(50)
        cnt, rank = np.array([_close(fl, p) for p in o.atoms()["x"]]).T
        if first is None and cnt.max() > 32:
            first = rank[cnt.argmax()]
        assert cnt.max() <= 64
    assert first >= 32 and (rank >= 32).any()
    assert len(o.mesh_contacts(2)["tag"]) > 0 and len(o.mesh_contacts(1)["tag"]) > 0


@pytest.mark.gpu
@pytest.mark.parametrize("walls", ["floor", "floor_first", "floor_last"])
def test_slots_grow_during_a_run(walls):
    import granb200
    sc = _scene(walls=walls)
    e, o = granb200.Engine(sc), oracle.Oracle(sc)
    e.setup()
    o.setup()
    total = np.zeros(len(_meshes(sc)), dtype=int)
    for _ in range(15):
        e.run(200)
        o.run(200)
        total += _check(e, o, sc)
    assert (total > 0).all()
    assert e.stats()["nbuilds"] == o.nbuilds > 3


@pytest.mark.gpu
@pytest.mark.parametrize("walls", ["floor", "floor_last"])
def test_slots_grow_at_a_restart(walls):
    """The restarted context lists 32 triangles an atom until its setup finds more."""
    import granb200
    from parity_util import restart_scenario
    sc = _scene(walls=walls)
    e, o = granb200.Engine(sc), oracle.Oracle(sc)
    e.setup()
    o.setup()
    e.run(3000)
    o.run(3000)
    sc2 = restart_scenario(sc, e.atoms())
    e2, o2 = granb200.Engine(sc2), oracle.Oracle(sc2)
    h = e.history()
    for x in (e2, o2):
        x.upload_history(h["npartner"], h["partner_tag"], h["hist"])
        for k in _meshes(sc):
            m = e.mesh_history(k)
            x.upload_mesh_hist(k, m["npartner"], m["tri"], m["hist"])
        x.setup()
    for k in _meshes(sc):
        assert mesh_contact_map(e2.mesh_contacts(k)) == mesh_contact_map(e.mesh_contacts(k)) != {}
    for _ in range(3):
        _check(e2, o2, sc)
        e2.run(200)
        o2.run(200)
