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
    assert ce["pairs_solved"] == co["pairs_solved"] and (ce["pairs_solved"] > 0 or n < 8)
    assert abs(ce["iters"] - co["iters"]) <= max(2, 0.01 * co["iters"])


SUMS = r"""
#include <cuda_runtime.h>
#include "gb2_mlp.cuh"
#include "gb2_sq_solve.cuh"
__global__ void k(const double *a, const double *b, double *s4, double *s8)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    s4[i] = gb2::sq::sum4(0xffffffffu, a[i] * 0.5, b[i]);   // a product the compiler could contract further
    s8[i] = gb2::sq::sum8(0xffffffffu, a[i], b[i]);
}
extern "C" int run(const double *a, const double *b, int n, double *s4, double *s8)
{
    double *d;
    if (cudaMalloc(&d, n * 32)) return 1;
    cudaMemcpy(d, a, n * 8, cudaMemcpyHostToDevice);
    cudaMemcpy(d + n, b, n * 8, cudaMemcpyHostToDevice);
    k<<<n / 128, 128>>>(d, d + n, d + 2 * n, d + 3 * n);
    cudaMemcpy(s4, d + 2 * n, n * 8, cudaMemcpyDeviceToHost);
    const int rc = cudaMemcpy(s8, d + 3 * n, n * 8, cudaMemcpyDeviceToHost) != cudaSuccess;
    cudaFree(d);
    return rc;
}
"""


def _contracted(a, b):
    """What a fused multiply-add in each lane's first butterfly step would give
    (own product unrounded, partner's rounded), by exact rational arithmetic."""
    from fractions import Fraction
    p = a * b
    own = [float(Fraction(x) * Fraction(y) + Fraction(q)) for x, y, q in zip(a, b, p.reshape(-1, 2)[:, ::-1].ravel())]
    return np.array(own)


def test_group_sums_are_the_same_in_every_lane(tmp_path):
    """The solver's control flow rests on it.  Built with the flags of the
    superquadric unit, contraction on: the contracted form differs between the
    two lanes of a pair for these operands (checked here on the host)."""
    import ctypes
    import subprocess
    csrc = os.path.join(HERE, "..", "liggghts-public_b200", "csrc")
    src, so = tmp_path / "t.cu", tmp_path / "t.so"
    src.write_text(SUMS)
    subprocess.run(["nvcc", "-O3", "-std=c++17", "-gencode", "arch=compute_100a,code=sm_100a", "-I", csrc, "-shared",
                    "-Xcompiler", "-fPIC", "-o", str(so), str(src)], check=True)
    lib, n = ctypes.CDLL(str(so)), 128 * 64
    rng = np.random.default_rng(11)
    a, b = (rng.uniform(-1, 1, n) * 10.0 ** rng.uniform(-6, 6, n) for _ in range(2))
    s4, s8 = np.empty(n), np.empty(n)
    P = lambda v: v.ctypes.data_as(ctypes.POINTER(ctypes.c_double))  # noqa: E731
    assert lib.run(P(a), P(b), n, P(s4), P(s8)) == 0
    def butterfly(p, lanes):
        p = p.reshape(-1, lanes)
        while p.shape[1] > 1:
            p = p[:, 0::2] + p[:, 1::2]
        return np.repeat(p[:, 0], lanes)
    assert np.array_equal(s4, butterfly((a * 0.5) * b, 4))
    assert np.array_equal(s8, butterfly(a * b, 8))
    c = _contracted(a[:512], b[:512]).reshape(-1, 2)
    assert (c[:, 0] != c[:, 1]).any()


def _aligned_boxes(n, blk, seed=5):
    """Particles of one orientation, faces nearly parallel and nearly flat, in slight overlap."""
    sc = S.sq_packing(n=n, seed=seed)
    a, rng = sc["atoms"], np.random.default_rng(seed + 1)
    a["blockiness"] = np.full(n, blk)
    a["quat"][:] = S.random_quaternions(rng, 1)[0]
    w, x, y, z = a["quat"][0]
    R = np.array([[w * w + x * x - y * y - z * z, 2 * (x * y - w * z), 2 * (x * z + w * y)],
                  [2 * (x * y + w * z), w * w - x * x + y * y - z * z, 2 * (y * z - w * x)],
                  [2 * (x * z - w * y), 2 * (y * z + w * x), w * w - x * x - y * y + z * z]])
    a["shape"][:] = 1.5e-3 * rng.uniform(0.8, 1.2, (n, 3))
    vol = S.sq_volume(a["shape"], a["blockiness"])
    a.update(rmass=vol * 2500.0, inertia=S.sq_inertia(a["shape"], a["blockiness"], 2500.0), volume=vol)
    m, i = int(np.ceil(n ** (1 / 3))), np.arange(n)
    g = np.stack([i % m, (i // m) % m, i // (m * m)], axis=1).astype(float)
    a["x"] = np.ascontiguousarray((g * 3e-3 * 0.97 + rng.uniform(-4e-4, 4e-4, (n, 3))) @ R.T)
    return sc


@pytest.mark.parametrize("blk,tol", [(4.0, 0.002), (8.0, 0.04), (12.0, 0.08)])
def test_flat_faces_take_the_oracles_iterations(blk, tol):
    """Where the Hessians are nearly singular the Newton steps have to be those of pivoted elimination, as in the
    oracle: the first contacts take its iterations (steps from cofactors alone took 8 % fewer at blockiness 8 and
    27 % fewer at 12, in the oracle's own arithmetic, and left more solves unconverged)."""
    import granb200
    sc = _aligned_boxes(64, blk)
    e, o = granb200.SqEngine(sc), oracle.SqOracle(sc)
    e.setup()
    o.setup()
    ce, co = e.counters(), o.counters()
    print(blk, ce, co)
    assert ce["pairs_solved"] == co["pairs_solved"] > 100 and ce["solves"] == co["solves"]
    assert abs(ce["iters"] - co["iters"]) <= tol * co["iters"]
