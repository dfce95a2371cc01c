"""Atoms with more than 64 list entries on a side: the counts at the edges of
the warp's chunks, on either side of the half list, bit for bit against the
oracle."""
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

pytestmark = pytest.mark.gpu


def _cluster(m, big_first, rolling):
    """One 3 mm sphere and m small ones on its surface, most of them touching it."""
    rng = np.random.default_rng(m)
    k = np.arange(m) + 0.5
    th, ph = np.arccos(1.0 - 2.0 * k / m), np.pi * (1.0 + 5 ** 0.5) * k
    d = np.stack([np.sin(th) * np.cos(ph), np.sin(th) * np.sin(ph), np.cos(th)], axis=1)
    small = 0.15e-3
    x = d * (3e-3 + small * (1.0 + rng.uniform(-0.02, 0.01, m)))[:, None]
    pos = np.concatenate([np.zeros((1, 3)), x]) if big_first else np.concatenate([x, np.zeros((1, 3))])
    rad = np.full(m + 1, small)
    rad[0 if big_first else m] = 3e-3
    sc = S.sphere_pour(n=m + 1, seed=1, box=(0.04, 0.04, 0.2))
    sc["atoms"] = S._atoms(pos + np.array([0.02, 0.02, 0.02]), rad, 2500.0, rng.uniform(-0.2, 0.2, (m + 1, 3)),
                           rng.uniform(-20.0, 20.0, (m + 1, 3)))
    sc.update(dt=2e-6, rolling_cdt=int(rolling), sortfreq=0)
    sc["rollfriction"] = np.array([[0.1]])
    return sc


@pytest.mark.parametrize("big_first", [True, False])
@pytest.mark.parametrize("m,rolling", [(60, True), (64, False), (65, True), (127, True), (128, False), (129, True),
                                       (200, True), (255, False)])
def test_long_lists_match_oracle(m, big_first, rolling):
    import granb200
    sc = _cluster(m, big_first, rolling)
    e, o = granb200.Engine(sc), oracle.Oracle(sc)
    e.setup()
    o.setup()
    for steps in (0, 1, 40):
        e.run(steps)
        o.run(steps)
        a, b = e.atoms(), o.atoms()
        for k in ("tag", "x", "v", "omega", "f", "torque"):
            assert np.array_equal(a[k], b[k]), (k, steps)
        p, q = e.pairs(), o.pairs()
        for k in ("tag_i", "tag_j", "flag", "hist"):
            assert np.array_equal(p[k], q[k]), (k, steps)
    assert (q["flag"] != 0).sum() > m // 3
