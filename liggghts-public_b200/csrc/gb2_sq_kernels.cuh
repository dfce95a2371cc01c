// gb2_sq_kernels.cuh -- kernels of the superquadric time step.
//
// Layout (structure of arrays, 32-byte records):
//   per atom: x {x, y, z, rbound}, v {vx, vy, vz, m}, q {w, i, j, k},
//             L {angmom, -}, w {omega, -}, f, t, shape {a, b, c, n},
//             inert {Ixx, Iyy, Izz, rvol}, xhold
//   half list in CSR form by owner i (neighbours j > i, ascending):
//             start[i] .. start[i+1], nbr[s]; per slot s the contact history
//             flag, state (far/close/intersect), cp {contact point, -},
//             alpha {alphaA, alphaB}, shear {s0, s1, s2, -}
//   per slot results of the pair pass: fi (force on i), ti, tj (torques)
//   reverse CSR by j: rstart[j] .. rstart[j+1], rslot[r] = slot index (ascending i)
#pragma once

#include "gb2_sq.cuh"
#include "gb2_internal.h"
#include "gb2_mma.cuh"

namespace gb2 {
namespace sq {

struct SqDev {
    int n;
    dbl4 *x, *v, *q, *L, *w, *f, *t, *shape, *inert, *xhold;
    // list
    int *start, *nbr, *flag, *state;
    dbl4 *cp, *shear;
    double2 *alpha;
    dbl4 *pfi, *pti, *ptj;
    int *rstart, *rslot;
    // physics
    double dt, skin, triggersq;
    double Yeff, Geff, betaeff, mu;
    // counters: iterations, solves, pairs solved, learned guesses used, learned guesses rejected
    unsigned long long *cnt;
    int *dflag;
    // steps queued ahead: the lowest step whose end asked for a rebuild of the
    // next one (null when not queuing), this launch's step, and a page-locked
    // host word set with it
    int *dstop;
    int step;
    volatile int *hstop;
    // learned initial guess (null when off)
    const float *mlp;
};

// One particle's state through the integrator
struct SqBody {
    dbl4 x, v;
    double q[4], L[3], w[3];
};

__device__ __forceinline__ bool sq_cancelled(const SqDev &D) { return D.dstop && *(volatile int *)D.dstop < D.step; }

// FixNVEAsphereBase::initial_integrate, integration_scheme 1
// (src/fix_nve_asphere_base.cpp:319-444) with force f and torque tq
__device__ __forceinline__ void sq_initial(const SqDev &D, SqBody &B, const dbl4 &f, const dbl4 &tq, const dbl4 &in4)
{
    const double dtv = D.dt, dtf = 0.5 * D.dt * 1.0, dtf2 = 2.0 * dtf, dtq = 0.5 * dtv;
    using namespace integrator;
    const double in[3] = {in4.x, in4.y, in4.z};
    double R[9], mbody[3], conjqm[4], tbody[3], fquat[4], wbody[3];
    integrator::quat_to_mat(B.q, R);
    const double dtfm = dtf / B.v.w;
    axpy(dtfm, f.x, B.v.x);
    axpy(dtfm, f.y, B.v.y);
    axpy(dtfm, f.z, B.v.z);
    axpy(dtv, B.v.x, B.x.x);
    axpy(dtv, B.v.y, B.x.y);
    axpy(dtv, B.v.z, B.x.z);
    const double Tv[3] = {tq.x, tq.y, tq.z};
    integrator::tmatvec(R, B.L, mbody);
    quatvec(B.q, mbody, conjqm);
    for (int k = 0; k < 4; k++) conjqm[k] *= 2.0;
    integrator::tmatvec(R, Tv, tbody);
    quatvec(B.q, tbody, fquat);
    for (int k = 0; k < 4; k++) axpy(dtf2, fquat[k], conjqm[k]);
    no_squish_rotate(3, conjqm, B.q, in, dtq);
    no_squish_rotate(2, conjqm, B.q, in, dtq);
    no_squish_rotate(1, conjqm, B.q, in, dtv);
    no_squish_rotate(2, conjqm, B.q, in, dtq);
    no_squish_rotate(3, conjqm, B.q, in, dtq);
    const double norm =
        1.0 / sqrt(add(sum3(mul(B.q[0], B.q[0]), mul(B.q[1], B.q[1]), mul(B.q[2], B.q[2])), mul(B.q[3], B.q[3])));
    for (int k = 0; k < 4; k++) B.q[k] *= norm;
    integrator::quat_to_mat(B.q, R);
    invquatvec(B.q, conjqm, mbody);
    for (int d = 0; d < 3; d++) mbody[d] *= 0.5;
    for (int d = 0; d < 3; d++) wbody[d] = mbody[d] / in[d];
    integrator::matvec(R, mbody, B.L);
    integrator::matvec(R, wbody, B.w);
}

// FixNVEAsphereBase::final_integrate, integration_scheme 1 (:523-620)
__device__ __forceinline__ void sq_final(const SqDev &D, SqBody &B, const dbl4 &f, const dbl4 &tq, const dbl4 &in4)
{
    const double dtf = 0.5 * D.dt * 1.0, dtf2 = dtf * 2.0;
    using namespace integrator;
    const double in[3] = {in4.x, in4.y, in4.z};
    double R[9], tbody[3], mbody[3], conjqm[4], fquat[4], wbody[3];
    const double dtfm = dtf / B.v.w;
    integrator::quat_to_mat(B.q, R);
    axpy(dtfm, f.x, B.v.x);
    axpy(dtfm, f.y, B.v.y);
    axpy(dtfm, f.z, B.v.z);
    const double Tv[3] = {tq.x, tq.y, tq.z};
    integrator::tmatvec(R, Tv, tbody);
    integrator::tmatvec(R, B.L, mbody);
    quatvec(B.q, mbody, conjqm);
    for (int k = 0; k < 4; k++) conjqm[k] *= 2.0;
    quatvec(B.q, tbody, fquat);
    for (int k = 0; k < 4; k++) axpy(dtf2, fquat[k], conjqm[k]);
    invquatvec(B.q, conjqm, mbody);
    for (int d = 0; d < 3; d++) mbody[d] *= 0.5;
    for (int d = 0; d < 3; d++) wbody[d] = mbody[d] / in[d];
    integrator::matvec(R, mbody, B.L);
    integrator::matvec(R, wbody, B.w);
}

__device__ __forceinline__ SqBody sq_load(const SqDev &D, int i)
{
    SqBody B;
    B.x = D.x[i];
    B.v = D.v[i];
    const dbl4 q = D.q[i], L = D.L[i];
    B.q[0] = q.x, B.q[1] = q.y, B.q[2] = q.z, B.q[3] = q.w;
    B.L[0] = L.x, B.L[1] = L.y, B.L[2] = L.z;
    return B;
}

__device__ __forceinline__ void sq_store(const SqDev &D, int i, const SqBody &B, bool moved)
{
    if (moved) {
        D.x[i] = B.x;
        D.q[i] = dbl4{B.q[0], B.q[1], B.q[2], B.q[3]};
    }
    D.v[i] = B.v;
    D.L[i] = dbl4{B.L[0], B.L[1], B.L[2], 0.0};
    D.w[i] = dbl4{B.w[0], B.w[1], B.w[2], 0.0};
}

// Neighbor::check_distance
__device__ __forceinline__ bool sq_far(const SqDev &D, int i, const dbl4 &x)
{
    const dbl4 h = D.xhold[i];
    const double dx = x.x - h.x, dy = x.y - h.y, dz = x.z - h.z;
    return dx * dx + dy * dy + dz * dz > D.triggersq;
}

// the first step of a run: initial_integrate and the displacement test
__global__ void k_sq_initial(SqDev D)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= D.n) return;
    SqBody B = sq_load(D, i);
    sq_initial(D, B, D.f[i], D.t[i], D.inert[i]);
    sq_store(D, i, B, true);
    if (sq_far(D, i, B.x)) *D.dflag = 1;
}

// omega from angular momentum (set-up)
__global__ void k_sq_omega(SqDev D)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= D.n) return;
    const dbl4 q4 = D.q[i], L4 = D.L[i], in4 = D.inert[i];
    const double q[4] = {q4.x, q4.y, q4.z, q4.w}, Lv[3] = {L4.x, L4.y, L4.z};
    double R[9], mb[3], wb[3], wo[3];
    quat_to_mat(q, R);
    tmatvec(R, Lv, mb);
    wb[0] = mb[0] / in4.x;
    wb[1] = mb[1] / in4.y;
    wb[2] = mb[2] / in4.z;
    matvec(R, wb, wo);
    D.w[i] = dbl4{wo[0], wo[1], wo[2], 0.0};
}

// ------------------------------------------------------------------
// learned initial guess: MLP 14 -> 64 -> 64 -> 64 -> 4 (ReLU), BF16 weights
// and activations with FP32 accumulation, parameters packed as
//   in_mean[14] in_std[14] out_mean[4] out_std[4]
//   W1[64][14] b1[64] W2[64][64] b2[64] W3[64][64] b3[64] W4[4][64] b4[4]
constexpr int kMlpIn = 14, kMlpH = 64, kMlpOut = 4;
constexpr int kMlpOffW1 = 36, kMlpOffB1 = kMlpOffW1 + kMlpH * kMlpIn, kMlpOffW2 = kMlpOffB1 + kMlpH,
              kMlpOffB2 = kMlpOffW2 + kMlpH * kMlpH, kMlpOffW3 = kMlpOffB2 + kMlpH,
              kMlpOffB3 = kMlpOffW3 + kMlpH * kMlpH, kMlpOffW4 = kMlpOffB3 + kMlpH,
              kMlpOffB4 = kMlpOffW4 + kMlpOut * kMlpH, kMlpSize = kMlpOffB4 + kMlpOut;

__device__ __forceinline__ float bf16_round(float x) { return __bfloat162float(__float2bfloat16_rn(x)); }

// pair features in particle i's body frame, lengths over s = ri + rj
// (ri = cbrt(abc)): centre of j (3), rotation vector of q_i^-1 q_j (3),
// half-axes of i and j (6), (n - 2) / 6 of i and j (2)
__device__ __forceinline__ double pair_features(const double *ci, const double *qi, const double *si, double ni,
                                                const double *cj, const double *qj, const double *sj, double nj,
                                                const double *Ri, float *feat)
{
    const double ri = cbrt(si[0] * si[1] * si[2]), rj = cbrt(sj[0] * sj[1] * sj[2]);
    const double s = ri + rj, sinv = 1.0 / s;
    const double d[3] = {cj[0] - ci[0], cj[1] - ci[1], cj[2] - ci[2]};
    double dl[3];
    tmatvec(Ri, d, dl);
    // q_rel = conj(q_i) * q_j
    const double a0 = qi[0], a1 = -qi[1], a2 = -qi[2], a3 = -qi[3];
    double r0 = a0 * qj[0] - a1 * qj[1] - a2 * qj[2] - a3 * qj[3];
    double r1 = a0 * qj[1] + qj[0] * a1 + a2 * qj[3] - a3 * qj[2];
    double r2 = a0 * qj[2] + qj[0] * a2 + a3 * qj[1] - a1 * qj[3];
    double r3 = a0 * qj[3] + qj[0] * a3 + a1 * qj[2] - a2 * qj[1];
    if (r0 < 0) {
        r0 = -r0;
        r1 = -r1;
        r2 = -r2;
        r3 = -r3;
    }
    const double vn = sqrt(r1 * r1 + r2 * r2 + r3 * r3);
    const double ang = 2.0 * atan2(vn, r0);
    const double k = vn > 0 ? ang / vn : 2.0;
    feat[0] = (float)(dl[0] * sinv);
    feat[1] = (float)(dl[1] * sinv);
    feat[2] = (float)(dl[2] * sinv);
    feat[3] = (float)(k * r1);
    feat[4] = (float)(k * r2);
    feat[5] = (float)(k * r3);
    for (int c = 0; c < 3; c++) {
        feat[6 + c] = (float)(si[c] * sinv);
        feat[9 + c] = (float)(sj[c] * sinv);
    }
    feat[12] = (float)((ni - 2.0) / 6.0);
    feat[13] = (float)((nj - 2.0) / 6.0);
    return s;
}

// Inference on the tensor cores.  The parameters are staged once per block
// (weights rounded to BF16 and zero-padded exactly as the training kernel
// does), and each warp runs the forward pass of its 32 lanes' pairs as two
// 16-row tiles through the training kernel's own layers (mma.sync m16n8k16,
// FP32 accumulation, bias + ReLU, BF16 activations), so a guess is computed
// with the arithmetic the network was trained with.
struct MlpInfer {
    __nv_bfloat16 W1[kMlpH][16], W2[kMlpH][kMlpH], W3[kMlpH][kMlpH], W4[8][kMlpH];
    float b1[kMlpH], b2[kMlpH], b3[kMlpH], b4[8];
    float stat[2 * kMlpIn + 2 * kMlpOut];   // in_mean, in_std, out_mean, out_std
    __nv_bfloat16 X[4][32][16];             // per warp: normalised features
    __nv_bfloat16 H[4][2][16][kMlpH];       // per warp: activations of one tile
    float Y[4][32][kMlpOut];                // per warp: outputs
};

// all threads of the block; the caller synchronises the block afterwards
__device__ __forceinline__ void mlp_stage(MlpInfer &S, const float *__restrict__ P)
{
    const int tid = threadIdx.x, nt = blockDim.x;
    for (int e = tid; e < kMlpH * 16; e += nt) {
        const int o = e / 16, c = e % 16;
        S.W1[o][c] = __float2bfloat16_rn(c < kMlpIn ? P[kMlpOffW1 + o * kMlpIn + c] : 0.f);
    }
    for (int e = tid; e < kMlpH * kMlpH; e += nt) {
        S.W2[e / kMlpH][e % kMlpH] = __float2bfloat16_rn(P[kMlpOffW2 + e]);
        S.W3[e / kMlpH][e % kMlpH] = __float2bfloat16_rn(P[kMlpOffW3 + e]);
    }
    for (int e = tid; e < 8 * kMlpH; e += nt) {
        const int o = e / kMlpH;
        S.W4[o][e % kMlpH] = __float2bfloat16_rn(o < kMlpOut ? P[kMlpOffW4 + e] : 0.f);
    }
    for (int e = tid; e < kMlpH; e += nt) {
        S.b1[e] = P[kMlpOffB1 + e];
        S.b2[e] = P[kMlpOffB2 + e];
        S.b3[e] = P[kMlpOffB3 + e];
    }
    if (tid < 8) S.b4[tid] = tid < kMlpOut ? P[kMlpOffB4 + tid] : 0.f;
    for (int e = tid; e < 2 * kMlpIn + 2 * kMlpOut; e += nt) S.stat[e] = P[e];
}

// The forward pass of the warp's 32 lanes (called by the whole warp of a
// 128-thread block; lanes with active false contribute zero rows): out =
// de-normalised (point in i's frame / s, mu) of the lane's pair.
__device__ __forceinline__ void mlp_infer_warp(MlpInfer &S, bool active, const float *feat, float *out)
{
    const int lane = threadIdx.x & 31, w = (threadIdx.x >> 5) & 3;
    for (int c = 0; c < 16; c++) {
        const float v = (active && c < kMlpIn) ? (feat[c] - S.stat[c]) / S.stat[kMlpIn + c] : 0.f;
        S.X[w][lane][c] = __float2bfloat16_rn(v);
    }
    __syncwarp();
    const int g = lane >> 2, t = lane & 3;
    for (int tile = 0; tile < 2; tile++) {
        layer_fwd<16, kMlpH>(&S.X[w][16 * tile][0], &S.W1[0][0], S.b1, &S.H[w][0][0][0], true);
        __syncwarp();
        layer_fwd<kMlpH, kMlpH>(&S.H[w][0][0][0], &S.W2[0][0], S.b2, &S.H[w][1][0][0], true);
        __syncwarp();
        layer_fwd<kMlpH, kMlpH>(&S.H[w][1][0][0], &S.W3[0][0], S.b3, &S.H[w][0][0][0], true);
        __syncwarp();
        float acc[4] = {0.f, 0.f, 0.f, 0.f};
        for (int k0 = 0; k0 < kMlpH; k0 += 16) {
            unsigned a[4], bb[2];
            load_a<false>(&S.H[w][0][0][0], kMlpH, 0, k0, a);
            load_b<true>(&S.W4[0][0], kMlpH, k0, 0, bb);
            mma16816(acc, a, bb);
        }
        for (int q = 0; q < 4; q++) {
            const int r = g + (q >> 1) * 8, c = 2 * t + (q & 1);
            if (c < kMlpOut) S.Y[w][16 * tile + r][c] = acc[q] + S.b4[c];
        }
        __syncwarp();
    }
    for (int c = 0; c < kMlpOut; c++)
        out[c] = S.Y[w][lane][c] * S.stat[2 * kMlpIn + kMlpOut + c] + S.stat[2 * kMlpIn + c];
    __syncwarp();
}

// Newton iterations granted to the solve from the learned guess.  A start
// the network places well converges in ~10; one that needs more is handed to
// the homotopy, whose result is the plain method's anyway, so the pairs that
// defeat both methods no longer pay the full iteration bound twice.
constexpr int kLearnedNewton = 48;

// Contact point of a pair without a previous point from the network's
// output `out` (point in i's frame / s, mu): one Newton solve of at most
// kLearnedNewton iterations.  The caller accepts it when it converged to
// merit < 1e-10 and otherwise runs the homotopy.
__device__ __forceinline__ void used_learned_guess(const float *out, const double *ci, const double *qi,
                                                   const double *si, double ni, const double *cj, const double *qj,
                                                   const double *sj, double nj, Newton &o, int &iters, int &solves)
{
    double Ri[9];
    quat_to_mat(qi, Ri);
    const double s = cbrt(si[0] * si[1] * si[2]) + cbrt(sj[0] * sj[1] * sj[2]);
    const double pl[3] = {out[0] * s, out[1] * s, out[2] * s};
    double g[3];
    matvec(Ri, pl, g);
    for (int k = 0; k < 3; k++) g[k] += ci[k];
    contact_point<kLearnedNewton>(ci, qi, si, ni, cj, qj, sj, nj, 1, g, true, (double)fabsf(out[3]), o, iters,
                                  solves);
}

// The network's features of a pair (i's body frame)
__device__ __forceinline__ void pair_features_of(const double *ci, const double *qi, const double *si, double ni,
                                                 const double *cj, const double *qj, const double *sj, double nj,
                                                 float *feat)
{
    double Ri[9];
    quat_to_mat(qi, Ri);
    pair_features(ci, qi, si, ni, cj, qj, sj, nj, Ri, feat);
}

// Contact point of a pair without a previous point in one call: the learned
// guess when the network's output is given, the homotopy when it is
// rejected or absent.  used: 1 learned guess accepted, -1 rejected, 0 off.
__device__ __forceinline__ void first_contact(const float *out, const double *ci, const double *qi, const double *si,
                                              double ni, const double *cj, const double *qj, const double *sj,
                                              double nj, Newton &o, int &iters, int &solves, int &used)
{
    used = 0;
    if (out) {
        int it1, sv1;
        used_learned_guess(out, ci, qi, si, ni, cj, qj, sj, nj, o, it1, sv1);
        if (!o.fail && o.merit < 1e-10) {
            iters = it1;
            solves = sv1;
            used = 1;
            return;
        }
        int it2, sv2;
        contact_point(ci, qi, si, ni, cj, qj, sj, nj, 0, nullptr, false, 0.0, o, it2, sv2);
        iters = it1 + it2;
        solves = sv1 + sv2;
        used = -1;
        return;
    }
    contact_point(ci, qi, si, ni, cj, qj, sj, nj, 0, nullptr, false, 0.0, o, iters, solves);
}

// ------------------------------------------------------------------
// pair pass (PairGran::compute with the superquadric surface model,
// src/pair_gran_base.h:255-430, src/surface_model_superquadric.h:108-205,
// non-spherical Hertz/history): k_sq_screen tests every half-list slot
// (bounding spheres, oriented boxes) and marks the slots that need a
// contact-point solve on one of two lists, first contacts and warm starts
// (a previous point exists);
// k_sq_solve (gb2_sq_solve.cuh) runs the solves, first contacts first: their
// chains, through the homotopy or the learned guess, are the longest, so they
// start at once and the short warm starts fill the GPU around them.  Every
// slot's result is the one-pass result (the solves are deterministic and
// independent).

// lists of one pair pass: 0 first contacts, 1 warm starts
struct SqWork {
    int *list[2];
    int *n;      // item counts, [2]; zeroed by the step's end (k_sq_advance)
    int *next;   // items taken (over both lists)
};

// every slot: no force unless a solve below finds a contact; the bounding
// spheres and (for a pair not yet intersecting) the oriented boxes decide
// whether the slot needs a solve and which kind, and a warp appends its slots
// to the two lists with one atomic each (the order of a list affects no
// result; two stable selections were four launches, ~15 us of a step)
__global__ void k_sq_screen(SqDev D, const int *__restrict__ own, int nslots, SqWork W)
{
    if (sq_cancelled(D)) return;
    const int sl = blockIdx.x * blockDim.x + threadIdx.x;
    int kind = -1;
    if (sl < nslots) {
        const int i = own[sl], j = D.nbr[sl];
        const dbl4 xi4 = D.x[i], xj4 = D.x[j];
        D.pfi[sl] = dbl4{0, 0, 0, 0};
        D.pti[sl] = dbl4{0, 0, 0, 0};
        D.ptj[sl] = dbl4{0, 0, 0, 0};
        const double dx = xi4.x - xj4.x, dy = xi4.y - xj4.y, dz = xi4.z - xj4.z;
        const double rsq = dx * dx + dy * dy + dz * dz, radsum = xi4.w + xj4.w;
        if (rsq < radsum * radsum) {
            const int state = D.state[sl];
            bool obb = true;
            if (state != INTERSECT) {
                const dbl4 qi4 = D.q[i], qj4 = D.q[j], si4 = D.shape[i], sj4 = D.shape[j];
                const double ci[3] = {xi4.x, xi4.y, xi4.z}, cj[3] = {xj4.x, xj4.y, xj4.z};
                const double qi[4] = {qi4.x, qi4.y, qi4.z, qi4.w}, qj[4] = {qj4.x, qj4.y, qj4.z, qj4.w};
                const double si[3] = {si4.x, si4.y, si4.z}, sj[3] = {sj4.x, sj4.y, sj4.z};
                double Ri[9], Rj[9];
                quat_to_mat(qi, Ri);
                quat_to_mat(qj, Rj);
                obb = obb_intersect(ci, Ri, si, cj, Rj, sj);
            }
            if (!obb) D.state[sl] = FAR;
            else kind = state == FAR ? 0 : 1;
        }
    }
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int l = 0; l < 2; l++) {
        const unsigned m = __ballot_sync(0xffffffffu, kind == l);
        if (!m) continue;
        int base = 0;
        if (lane == __ffs(m) - 1) base = atomicAdd(&W.n[l], __popc(m));
        base = __shfl_sync(0xffffffffu, base, __ffs(m) - 1);
        if (kind == l) W.list[l][base + __popc(m & ((1u << lane) - 1u))] = sl;
    }
}

// per-atom sums in the reference's order: slots where the atom is the j
// side (ascending i), then its own slots
__device__ __forceinline__ void sq_sums(const SqDev &D, int k, dbl4 &Fo, dbl4 &To)
{
    double F[3] = {0, 0, 0}, T[3] = {0, 0, 0};
    for (int r = D.rstart[k]; r < D.rstart[k + 1]; r++) {
        const int sl = D.rslot[r];
        const dbl4 f = D.pfi[sl];
        if (f.w == 0.0) continue;
        const dbl4 t = D.ptj[sl];
        F[0] += -f.x;
        F[1] += -f.y;
        F[2] += -f.z;
        T[0] += t.x;
        T[1] += t.y;
        T[2] += t.z;
    }
    for (int sl = D.start[k]; sl < D.start[k + 1]; sl++) {
        const dbl4 f = D.pfi[sl];
        if (f.w == 0.0) continue;
        const dbl4 t = D.pti[sl];
        F[0] += f.x;
        F[1] += f.y;
        F[2] += f.z;
        T[0] += t.x;
        T[1] += t.y;
        T[2] += t.z;
    }
    Fo = dbl4{F[0], F[1], F[2], 0.0};
    To = dbl4{T[0], T[1], T[2], 0.0};
}

// The end of a pair pass: the sums and, on a step (integrate), final_integrate
// and -- when the run continues (next) -- the next step's initial_integrate
// with its displacement test, per particle in one kernel: three kernels each
// read and wrote the same records.  Leaves the work lists empty for the next
// pass.
__global__ void k_sq_advance(SqDev D, SqWork W, int integrate, int next)
{
    if (sq_cancelled(D)) return;
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < 3) W.n[i] = 0;   // n[2] and next, which follows them
    if (i >= D.n) return;
    dbl4 f, t;
    sq_sums(D, i, f, t);
    D.f[i] = f;
    D.t[i] = t;
    if (!integrate) return;
    const dbl4 in4 = D.inert[i];
    SqBody B = sq_load(D, i);
    sq_final(D, B, f, t, in4);
    if (next) {
        sq_initial(D, B, f, t, in4);
        if (sq_far(D, i, B.x)) {
            *D.dflag = 1;
            if (D.dstop) {
                atomicMin(D.dstop, D.step);
                *D.hstop = 1;
            }
        }
    }
    sq_store(D, i, B, next != 0);
}

}  // namespace sq
}  // namespace gb2
