"""Both forms of the FP64 pair step, one lane per atom and two, on scenes of
any size: contexts of few atoms take two lanes and large ones one, so each
form is fixed here (GB2_PAIR_LANES) and compared with the reference's digests
bit for bit -- rolling friction, several atom types, periodic images, moving
meshes, insertion, and the mask enumeration of warps whose lists overflow."""
import pytest

import gb2_scenarios as S
import oracle
from parity_util import assert_atoms_equal, assert_mesh_equal, assert_pairs_equal
from ref_scenes import ALL_SCENES
from test_reference_parity import _compare, _run_checkpoints

pytestmark = pytest.mark.gpu
LARGE = ("config1_pour_20k_20000steps", "config2_hopper_1M_100steps")   # run in the form their size takes


def _digests(name):
    import granb200
    build, segments = ALL_SCENES[name]
    sc = build()
    e = granb200.Engine(sc)
    _compare(name, _run_checkpoints(e, sc, segments, lambda s: s.stats()["nbuilds"]))
    e.close()


@pytest.mark.parametrize("name", sorted(set(ALL_SCENES) - set(LARGE)))
def test_one_lane_matches_reference(name, monkeypatch):
    monkeypatch.setenv("GB2_PAIR_LANES", "1")
    _digests(name)


@pytest.mark.parametrize("name", ["hopper_packed_discharge", "bidisperse_long_lists", "insert_pack_periodic"])
def test_one_lane_mask_rounds_match_reference(name, monkeypatch):
    monkeypatch.setenv("GB2_PAIR_LANES", "1")
    monkeypatch.setenv("GB2_ITEM_CAP", "0")
    _digests(name)


@pytest.mark.parametrize("lanes", ["1", "2"])
@pytest.mark.parametrize("types,rolling", [(1, 1), (2, 0), (2, 1)])
def test_lanes_match_oracle_over_types(lanes, types, rolling, monkeypatch):
    """Material constants from the launch (one type) or the table, rolling friction on and off, a rotating mesh."""
    import granb200
    import numpy as np
    monkeypatch.setenv("GB2_PAIR_LANES", lanes)
    sc = S.drum(n=1500, diameter=0.05, length=0.03, n_theta=48, n_ax=12, cap_rings=3, omega=50.0, clearance=0.3e-3,
                vmax=0.05)
    n = len(sc["atoms"]["tag"])
    sc.update(sortfreq=200, rolling_cdt=rolling)
    if types == 2:
        sc["atoms"]["type"] = np.where(np.arange(n) % 3 == 0, 2, 1).astype(np.int32)
        sc.update(ntypes=2, youngs=np.array([5e6, 2e7]), poisson=np.array([0.45, 0.3]),
                  restitution=np.array([[0.3, 0.5], [0.5, 0.7]]), friction=np.array([[0.5, 0.2], [0.2, 0.4]]))
    sc["rollfriction"] = np.full((types, types), 0.1) + 0.1 * np.eye(types)
    e, o = granb200.Engine(sc), oracle.Oracle(sc)
    e.setup()
    o.setup()
    for _ in range(3):
        e.run(400)
        o.run(400)
        assert_atoms_equal(e, o)
        npairs, ntouch = assert_pairs_equal(e, o)
        assert_mesh_equal(e, o, 1)
    assert ntouch > 100
