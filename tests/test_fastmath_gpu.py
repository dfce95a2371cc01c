"""The branch-free FP64 quotients and roots (gb2_fastmath.cuh) against the
IEEE operations: random operands over the range the callers check, significands
near one and near all ones, and -- for the roots -- the radicands whose root
lies closest to a midpoint of two FP64 numbers.  Equal bit for bit."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
CSRC = os.path.join(os.path.dirname(os.path.abspath(__file__)), "..", "liggghts-public_b200", "csrc")

SRC = r"""
#include "gb2_fastmath.cuh"
using namespace gb2;
// counts, per operation, the operands whose results differ from the operators'
__global__ void k(const double *a, const double *b, int n, unsigned long long *bad)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    double y;
    const double x = a[i], d = b[i], s = fast_sqrt(x, y), t = sqrt(x);
    auto differ = [](double u, double v) { return __double_as_longlong(u) != __double_as_longlong(v); };
    if (differ(s, t)) atomicAdd(&bad[0], 1ull);
    if (fast_divisor(d)) {
        if (differ(fast_rcp(d), 1.0 / d)) atomicAdd(&bad[1], 1ull);
        if (differ(fast_div(x, d), x / d)) atomicAdd(&bad[2], 1ull);
        if (differ(fast_div(-x, d), -x / d)) atomicAdd(&bad[2], 1ull);
    }
    if (fast_divisor(t) && differ(fast_rcp_from(t, y), 1.0 / t)) atomicAdd(&bad[3], 1ull);
}
extern "C" int run(const double *a, const double *b, int n, unsigned long long *bad)
{
    double *da, *db;
    unsigned long long *dbad;
    if (cudaMalloc(&da, n * 8) || cudaMalloc(&db, n * 8) || cudaMalloc(&dbad, 32) || cudaMemset(dbad, 0, 32)) return 1;
    cudaMemcpy(da, a, n * 8, cudaMemcpyHostToDevice);
    cudaMemcpy(db, b, n * 8, cudaMemcpyHostToDevice);
    k<<<(n + 127) / 128, 128>>>(da, db, n, dbad);
    const int rc = cudaMemcpy(bad, dbad, 32, cudaMemcpyDeviceToHost) != cudaSuccess;
    cudaFree(da);
    cudaFree(db);
    cudaFree(dbad);
    return rc;
}
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    d = tmp_path_factory.mktemp("fastmath")
    src, so = d / "t.cu", d / "t.so"
    src.write_text(SRC)
    subprocess.run(["nvcc", "-O3", "-std=c++17", "-gencode", "arch=compute_100a,code=sm_100a", "--fmad=false", "-I", CSRC,
                    "-shared", "-Xcompiler", "-fPIC", "-o", str(so), str(src)], check=True)
    return ctypes.CDLL(str(so))


def _hard_radicands():
    """a in [1, 4) with a close to a midpoint's square.  A midpoint is k 2^-53
    in [1, 2), k odd with 54 bits; its square is k^2 2^-106.  a is a multiple of
    2^-52 in [1, 2) and of 2^-51 in [2, 4), so k^2 = c mod 2^54 (2^55) with a
    small c = 1 mod 8: the roots of c, four of them, by lifting."""
    out = []
    for bits in (54, 55):
        for c in range(-511, 513, 8):
            r = next(x for x in (1, 3, 5, 7) if (x * x - c) % 16 in (0, 8))
            for m in range(4, bits + 1):   # r^2 = c mod 2^m
                if (r * r - c) % (1 << m):
                    r += 1 << (m - 2)
            if (r * r - c) % (1 << bits):
                continue
            for k in {r, -r, r + (1 << (bits - 1)), -r + (1 << (bits - 1))}:
                k %= 1 << bits
                for kk in (k, k + (1 << bits)):
                    if not (1 << 53) <= kk < (1 << 54):
                        continue
                    a, shift = kk * kk - c, 106 - (52 if bits == 54 else 51)
                    v = a >> (106 - (52 if bits == 54 else 51))
                    assert v << shift == a
                    if v < (1 << 53):
                        out.append(v * 2.0 ** (-52 if bits == 54 else -51))
    return np.array(sorted(set(out)))


def _count(lib, a, b):
    a, b = np.ascontiguousarray(a), np.ascontiguousarray(b)
    bad = (ctypes.c_ulonglong * 4)()
    D = ctypes.POINTER(ctypes.c_double)
    assert lib.run(a.ctypes.data_as(D), b.ctypes.data_as(D), len(a), bad) == 0
    return list(bad)


@pytest.mark.parametrize("kind", ["random", "near_one", "near_all_ones", "hard_roots"])
def test_equal_to_the_ieee_operations(lib, kind):
    rng = np.random.default_rng(7)
    n = 4_000_000
    if kind == "hard_roots":
        h = _hard_radicands()
        assert len(h) > 100
        a = np.concatenate([h * 4.0 ** e for e in (-100, -31, 0, 1, 17, 99)])
        assert _count(lib, a, np.ones(len(a)) * 3.0)[0] == 0
        return
    def operands():
        m = rng.integers(0, 1 << 52, n, dtype=np.uint64)
        if kind == "near_one":
            m >>= rng.integers(20, 52, n, dtype=np.uint64)
        if kind == "near_all_ones":
            m = np.uint64((1 << 52) - 1) - (m >> rng.integers(20, 52, n, dtype=np.uint64))
        e = rng.integers(1023 - 200, 1023 + 200, n, dtype=np.uint64)
        return (m | (e << np.uint64(52))).view(np.float64)
    assert _count(lib, operands(), operands()) == [0, 0, 0, 0]
