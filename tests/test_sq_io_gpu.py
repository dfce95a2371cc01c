"""Superquadric upload and download on the device: odd counts, the check's
verdict (first bad particle, context untouched), partial downloads."""
import ctypes
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

pytestmark = pytest.mark.gpu
D = ctypes.POINTER(ctypes.c_double)


def _ptr(a):
    return a.ctypes.data_as(D)


@pytest.mark.parametrize("n", [1, 2, 127, 128, 129, 1001])
def test_upload_comes_back(n):
    import granb200
    sc = S.sq_packing(n=n, seed=n)
    e = granb200.SqEngine(sc)
    a = e.atoms()
    for k in ("x", "v", "quat", "angmom"):
        assert np.array_equal(a[k], sc["atoms"][k]), k
    q = np.zeros((n, 4))
    e._check(e.L.gb2_sq_download(e.h, n, None, None, _ptr(q), None, None, None, None))
    assert np.array_equal(q, sc["atoms"]["quat"])
    assert e.L.gb2_sq_download(e.h, n - 1, None, None, _ptr(q), None, None, None, None) != 0


def test_bad_particle_is_named_and_nothing_changes():
    import granb200
    sc = S.sq_packing(n=200, seed=5)
    e = granb200.SqEngine(sc)
    e.setup()
    e.run(3)
    before = e.atoms()
    for key, bad in (("blockiness", 1.9), ("rmass", 0.0), ("volume", float("nan"))):
        a = {k: v.copy() for k, v in sc["atoms"].items()}
        a[key][150] = a[key][37] = bad
        with pytest.raises(granb200.GB2Error, match="superquadric 37:"):
            granb200.SqEngine(dict(sc, atoms=a))
        keep = [np.ascontiguousarray(a[k]) for k in
                ("x", "v", "quat", "angmom", "shape", "blockiness", "rmass", "inertia", "volume")]
        assert e.L.gb2_sq_upload(e.h, 200, *[_ptr(k) for k in keep]) != 0
    after = e.atoms()
    for k in before:
        assert np.array_equal(before[k], after[k]), k
    e.run(3)   # still set up
