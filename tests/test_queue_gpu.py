"""Runs that end within a few steps of a rebuild request, where the queued
steps after the request are undone: bit for bit the states, contacts and
rebuild counts of a context that decides every step on the host
(GB2_QUEUE_DEPTH=0), over the same run lengths."""
import numpy as np
import pytest

import gb2_scenarios as S
from parity_util import assert_atoms_equal, assert_mesh_equal, assert_pairs_equal

pytestmark = pytest.mark.gpu


def _engine(sc, monkeypatch, depth):
    import granb200
    with monkeypatch.context() as m:
        if depth is None:
            m.delenv("GB2_QUEUE_DEPTH", raising=False)
        else:
            m.setenv("GB2_QUEUE_DEPTH", str(depth))
        e = granb200.Engine(sc)
    e.setup()
    return e


def _build_steps(e, n):
    """The steps 1..n on which e rebuilds, one step a run."""
    out, last = [], e.stats()["nbuilds"]
    for s in range(1, n + 1):
        e.run(1)
        now = e.stats()["nbuilds"]
        if now != last:
            out.append(s)
        last = now
    return out


def _segments(ends):
    ends = sorted(set(ends))
    return [b - a for a, b in zip([0] + ends[:-1], ends)]


def test_mesh_asks_on_the_last_step(monkeypatch):
    """A turning drum whose nodes move furthest: a run ends on the step on which the mesh asks, and the next one,
    of a single step, has to rebuild."""
    sc = S.drum(n=800, diameter=0.05, length=0.03, n_theta=48, n_ax=12, cap_rings=3, omega=50.0, clearance=0.3e-3,
                vmax=0.3)
    builds = _build_steps(_engine(sc, monkeypatch, 0), 600)
    assert len(builds) > 10 and min(np.diff(builds)) > 3
    q, r = _engine(sc, monkeypatch, None), _engine(sc, monkeypatch, 0)
    contacts = 0
    for n in _segments([b - 1 for b in builds[1:]] + builds[1:]):
        q.run(n)
        r.run(n)
        assert q.stats()["nbuilds"] == r.stats()["nbuilds"]
        assert_atoms_equal(q, r)
        assert_pairs_equal(q, r)
        contacts += assert_mesh_equal(q, r, 1)
        qn, rn = q.mesh_nodes(1), r.mesh_nodes(1)
        assert np.array_equal(qn[0], rn[0]) and np.array_equal(qn[1], rn[1])
    assert contacts > 0


@pytest.mark.parametrize("after", [1, 2, 3, 4, 5])
def test_stream_run_ends_after_a_request(monkeypatch, after):
    """Particles that fix insert/stream holds, pushed into free ones below its face; every run ends `after` steps
    after a step that asked for a rebuild."""
    sc = S.stream_pour(n_bed=200)
    x = sc["atoms"]["x"]
    x[:60, 2] = 0.0385 + 0.5e-3 * (np.arange(60) % 3)
    builds = [b for b in _build_steps(_engine(sc, monkeypatch, 0), 320)]
    asked = [b - 1 for b in builds if (b - 1) % 200 > 5]
    q, r = _engine(sc, monkeypatch, None), _engine(sc, monkeypatch, 0)
    held = 0
    for n in _segments([a + after for a in asked if a > 8]):
        q.run(n)
        r.run(n)
        assert q.stats()["nbuilds"] == r.stats()["nbuilds"]
        assert_atoms_equal(q, r)
        assert_pairs_equal(q, r)
        held += 1
    assert held > 5 and len(q.atoms()["x"]) > 200
