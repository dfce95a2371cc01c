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


CONTACT = r"""
#include "gb2_contact.cuh"
using namespace gb2;
// one contact per thread, by the branch-free form and by the operators:
// count[0] contacts the branch-free form refused, count[1] differing results,
// count[2] contacts that slide
__global__ void k(const double *in, int n, MatPair M, double dt, unsigned long long *count)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    double v[20];
    for (int c = 0; c < 20; c++) v[c] = in[(size_t)c * n + i];
    const double *d = v, *vi = v + 3, *vj = v + 6, *wi = v + 9, *wj = v + 12;
    const double rsq = d[0] * d[0] + d[1] * d[1] + d[2] * d[2], r = 1e-3, m = 1e-5;
    double s1[3] = {v[15], v[16], v[17]}, s2[3] = {v[15], v[16], v[17]};
    ContactOut a, b;
    const bool ok = pair_contact_fast(M, d[0], d[1], d[2], rsq, r, r, vi, vj, wi, wj, m, m, s1, true, dt, true, true, a);
    pair_contact<false>(M, d[0], d[1], d[2], rsq, r, r, vi, vj, wi, wj, m, m, s2, true, dt, true, true, b);
    bool same = true;
    for (int c = 0; c < 3; c++)
        same = same && __double_as_longlong(a.F[c]) == __double_as_longlong(b.F[c]) &&
               __double_as_longlong(a.T[c]) == __double_as_longlong(b.T[c]) &&
               __double_as_longlong(s1[c]) == __double_as_longlong(s2[c]);
    if (!ok) atomicAdd(&count[0], 1ull);
    if (ok && !same) atomicAdd(&count[1], 1ull);
    const double t = v[15] + v[16] + v[17], u = s2[0] + s2[1] + s2[2];
    if (fabs(u) < 0.9 * fabs(t)) atomicAdd(&count[2], 1ull);
}
extern "C" int run(const double *in, int n, double mu, unsigned long long *count)
{
    MatPair M;
    M.Yeff = 3e6, M.Geff = 1e6, M.betaeff = -0.2, M.mu = mu, M.mur = 0.1;
    M.Y2 = 2. * M.Yeff, M.G8 = 8. * M.Geff, M.Y43 = 4. / 3. * M.Yeff, M.b56 = -2. * GB2_SQRT_FIVE_OVER_SIX * M.betaeff;
    M.fast = 1;
    double *d;
    unsigned long long *c;
    if (cudaMalloc(&d, (size_t)n * 160) || cudaMalloc(&c, 24) || cudaMemset(c, 0, 24)) return 1;
    cudaMemcpy(d, in, (size_t)n * 160, cudaMemcpyHostToDevice);
    k<<<(n + 127) / 128, 128>>>(d, n, M, 1e-5, c);
    const int rc = cudaMemcpy(count, c, 24, cudaMemcpyDeviceToHost) != cudaSuccess;
    cudaFree(d);
    cudaFree(c);
    return rc;
}
"""


@pytest.fixture(scope="module")
def contact_lib(tmp_path_factory):
    d = tmp_path_factory.mktemp("contact")
    src, so = d / "t.cu", d / "t.so"
    src.write_text(CONTACT)
    subprocess.run(["nvcc", "-O3", "-std=c++17", "-gencode", "arch=compute_100a,code=sm_100a", "--fmad=false", "-I", CSRC,
                    "-shared", "-Xcompiler", "-fPIC", "-o", str(so), str(src)], check=True)
    return ctypes.CDLL(str(so))


@pytest.mark.parametrize("mu", [0.4, 0.0])
@pytest.mark.parametrize("zero", [(), (2,), (1, 2), (0, 1), "minus"])
def test_sliding_contacts_with_zero_components(contact_lib, zero, mu):
    """Sliding contacts in a plane, along an axis, or in general: none is refused, each equals the operators' result
    bit for bit, the signs of zeros included."""
    rng = np.random.default_rng(5)
    n = 100_000
    d = rng.normal(size=(n, 3))
    planar = list(zero) if zero != "minus" else [1]
    d[:, planar] = 0.0
    d *= (2e-3 * rng.uniform(0.97, 0.999, n) / np.linalg.norm(d, axis=1))[:, None]
    vec = [rng.uniform(-1, 1, (n, 3)) for _ in range(2)] + [rng.uniform(-50, 50, (n, 3)) for _ in range(2)]
    shear = rng.uniform(0.5, 1.0, (n, 3)) * rng.choice([-1.0, 1.0], (n, 3)) * 1e-2
    for c in planar:
        z = -0.0 if zero == "minus" else 0.0
        for a in vec[:2] + [shear]:
            a[:, c] = z
        for k in range(3):   # rotation about the plane's normal only
            if k != c:
                for a in vec[2:]:
                    a[:, k] = z
    cols = np.concatenate([d] + vec + [shear, np.zeros((n, 2))], axis=1).T
    cols = np.ascontiguousarray(cols)
    count = (ctypes.c_ulonglong * 3)()
    contact_lib.run.argtypes = [ctypes.POINTER(ctypes.c_double), ctypes.c_int, ctypes.c_double, ctypes.c_void_p]
    assert contact_lib.run(cols.ctypes.data_as(ctypes.POINTER(ctypes.c_double)), n, mu, count) == 0
    assert count[0] == 0 and count[1] == 0 and count[2] > n // 2, list(count)
