"""The atom sort over the bin sizes a caller may choose (sort_binsize): wider
and finer than the default, where the order comes from a sort of the bin keys
instead of counting.  The order, and with it every bit of a run, is the
oracle's; a few crowded bins cost a sort, not a pass per atom over its bin."""
import time

import numpy as np
import pytest

import gb2_scenarios as S
import oracle
from parity_util import assert_atoms_equal, assert_pairs_equal

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,binsize", [(1, 0.0), (1, 0.02), (700, 0.0), (700, 0.0013), (700, 0.004), (700, 0.0101),
                                       (700, 0.02), (700, 1e-4)])
def test_order_matches_oracle(n, binsize):
    import granb200
    sc = S.sphere_pour(n=n, seed=3, vmax=0.5, box=(0.02, 0.02, 0.2))
    sc.update(sortfreq=40, sortbinsize=binsize)
    e, o = granb200.Engine(sc), oracle.Oracle(sc)
    e.setup()
    o.setup()
    assert_atoms_equal(e, o)
    for _ in range(2):
        e.run(150)
        o.run(150)
        assert_atoms_equal(e, o)
        assert_pairs_equal(e, o)


def test_crowded_bins_are_sorted():
    """2M spheres in 16 sort bins, up to 225,000 each, against bins of the default size: the setup, which sorts
    once."""
    import granb200
    sc = S.sphere_pour(n=2_000_000, seed=3, box=(0.3, 0.3, 0.6))
    t = {}
    for binsize in (0.0, 0.15):
        sc["sortbinsize"] = binsize
        best = np.inf
        for _ in range(3):
            e = granb200.Engine(sc)
            e.sync()
            t0 = time.perf_counter()
            e.setup()
            e.sync()
            best = min(best, time.perf_counter() - t0)
            e.close()
        t[binsize] = best
    print(t)
    assert t[0.15] < 2 * t[0.0] + 0.01, t
