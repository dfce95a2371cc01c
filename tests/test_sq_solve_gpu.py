"""The cooperative contact-point solves at the sizes and shapes where their
groups can go wrong: fewer pairs than a warp has groups, counts that leave
groups idle or make them take several items, ellipsoids (the closed-form
overlap), integer and half-integer exponents, and a mixture of them -- against
the CPU oracle."""
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


@pytest.mark.parametrize("n,blk", [(2, None), (8, None), (27, "two"), (125, "integer"), (125, "half"), (216, "mixed"),
                                   (1000, None)])
def test_solves_match_oracle(n, blk):
    import granb200
    sc = S.sq_packing(n=n, seed=41 + n, fill=0.68)
    rng = np.random.default_rng(n)
    a = sc["atoms"]
    if blk is not None:
        choice = {"two": [2.0], "integer": [3.0, 4.0, 7.0], "half": [2.5, 3.5, 5.5],
                  "mixed": [2.0, 2.005, 3.0, 3.995, 4.5, 6.3, 8.0]}[blk]
        a["blockiness"] = rng.choice(choice, n)
        vol = S.sq_volume(a["shape"], a["blockiness"])
        a.update(rmass=vol * 2500.0, inertia=S.sq_inertia(a["shape"], a["blockiness"], 2500.0), volume=vol)
    e, o = granb200.SqEngine(sc), oracle.SqOracle(sc)
    e.setup()
    o.setup()
    for steps in (0, 20):
        e.run(steps)
        o.run(steps)
        p, q = e.pairs(), o.pairs()
        assert np.array_equal(p["tag_i"], q["tag_i"]) and np.array_equal(p["tag_j"], q["tag_j"])
        assert np.array_equal(p["state"], q["state"])
        live = q["state"] > 0
        # the oracle's own bars: contact points within 1e-9 of the particle size, forces within 1e-5 of the largest
        if live.any():
            assert np.abs(p["cp"][live] - q["cp"][live]).max() <= 1e-12
        f, g = e.atoms(), o.atoms()
        for k in ("f", "torque"):
            assert np.abs(f[k] - g[k]).max() <= 1e-5 * max(np.abs(g[k]).max(), 1e-30)
    ce, co = e.counters(), o.counters()
    assert ce["pairs_solved"] == co["pairs_solved"] and ce["pairs_solved"] > 0 or n < 8
    assert abs(ce["iters"] - co["iters"]) <= max(2, 0.01 * co["iters"])
