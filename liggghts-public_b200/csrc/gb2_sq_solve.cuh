// gb2_sq_solve.cuh -- the contact-point solves of one superquadric pair pass.
//
// Eight lanes solve one pair: lane 4 b + a evaluates axis a (0..2) of body b
// (lane 3 of each half adds zeros), so the six powers of a shape function
// evaluation -- the arithmetic of a solve -- run side by side, one per lane,
// and the value, gradient and Hessian sums are shuffles.  The scalars of the
// solve are replicated in the eight lanes: the butterfly sums round every
// product and every sum by itself, so they are the same in each lane bit for
// bit.  Control flow is uniform in a group by construction: what a group does
// next is decided by its first lane and taken from it by the others, so its
// shuffles and barriers are reached by all eight lanes whatever the compiler
// makes of the replicated arithmetic.
//
// What bounds it: a step holds few solves (27k among 1M slots of a 200k
// packing) and the longest chain -- a first contact's homotopy, 11 stages and
// up to ~100 Newton iterations, each with its golden-section search -- sets
// the time.  One thread per solve left the chip to a few latency-bound
// warps, each as slow as its slowest lane.  Here every trip of a warp's loop
// performs exactly one evaluation for each of its four groups, whatever state
// each is in (a start, a Newton trial, a golden-section point, a point of the
// line search that measures the overlap), and a group whose item is finished
// takes the next one, so no group waits for another.  A step of a 200,000
// particle packing (20 steps, ~22,000 solves each) went from 2.27 ms to
// 0.52 ms, one of 2,000 particles (60 steps) from 0.67 ms to 0.17 ms, with the
// same iteration and solve counts.  168 registers (3 blocks per SM) keep the
// state of a solve out of local memory but for some 25 doubles; a group of 16
// lanes would only shorten the golden-section pairs.
#pragma once

#include "gb2_sq_kernels.cuh"

namespace gb2 {
namespace sq {

// What a group evaluates next.
enum : int { Q_IDLE, Q_INIT1, Q_INIT2, Q_TRIAL, Q_GOLD_A, Q_GOLD_B, Q_GOLD_TAKE, Q_LINE, Q_DONE };

// a^b for a >= 0 and 0 <= b, by squaring with the set bits selected (no
// branch on b for b < 8, so lanes with different exponents stay together)
__device__ __forceinline__ double ipow(double a, int b)
{
    const double a2 = a * a, a4 = a2 * a2;
    double r = ((b & 1) ? a : 1.0) * ((b & 2) ? a2 : 1.0) * ((b & 4) ? a4 : 1.0);
    if (b >= 8) {
        double s = a4 * a4;
        for (int m = b >> 3; m; m >>= 1) {
            if (m & 1) r *= s;
            s *= s;
        }
    }
    return r;
}

// pow_abs() for a base >= 0 and an exponent >= 0
__device__ __forceinline__ double pow_pos(double base, double e)
{
    const double tol = 1e-12;
    if (e < tol || fabs(base - 1.0) < tol) return 1.0;
    if (base < tol) return 0.0;
    const double n = floor(e), nd = e - n;
    double r = ipow(base, (int)n);
    if (nd > 0.0) r *= fabs(2.0 * nd - 1.0) < 2.0 * tol ? sqrt(base) : pow(base, nd);
    return r;
}

// The Newton step: H x + c x4 = f, d.x = f4, with H symmetric (h: xx, xy, xz,
// yy, yz, zz), by the cofactors of the bordered matrix,
//   x = (f4 adj(H) c - d x (H (c x f))) / D,  x4 = (adj(H) d . f - det(H) f4) / D,
//   D = d . adj(H) c  (minus the determinant of the 4x4 matrix),
// which also holds for a singular H.  One division ends a chain of a dozen
// multiply-adds; elimination with partial pivoting was four of each in
// sequence, half of a trip's latency.  Where H is nearly singular -- flat faces
// at high blockiness -- the cofactors cancel, so the caller checks what the
// result leaves of each equation (row_met) and eliminates with pivoting
// (solve_pivoted) where that is not small.
__device__ __forceinline__ void solve_bordered(const double *h, const double *c, const double *d, const double *f,
                                               double f4, double *x)
{
    const double axx = h[3] * h[5] - h[4] * h[4], axy = h[2] * h[4] - h[1] * h[5], axz = h[1] * h[4] - h[2] * h[3];
    const double ayy = h[0] * h[5] - h[2] * h[2], ayz = h[1] * h[2] - h[0] * h[4], azz = h[0] * h[3] - h[1] * h[1];
    const double z[3] = {axx * c[0] + axy * c[1] + axz * c[2], axy * c[0] + ayy * c[1] + ayz * c[2],
                         axz * c[0] + ayz * c[1] + azz * c[2]};
    const double w[3] = {axx * d[0] + axy * d[1] + axz * d[2], axy * d[0] + ayy * d[1] + ayz * d[2],
                         axz * d[0] + ayz * d[1] + azz * d[2]};
    const double det = h[0] * axx + h[1] * axy + h[2] * axz;
    double cf[3], r[3];
    cross3(c, f, cf);
    const double hv[3] = {h[0] * cf[0] + h[1] * cf[1] + h[2] * cf[2], h[1] * cf[0] + h[3] * cf[1] + h[4] * cf[2],
                          h[2] * cf[0] + h[4] * cf[1] + h[5] * cf[2]};
    cross3(d, hv, r);
    const double D = dot3(d, z), inv = 1.0 / D;
    for (int k = 0; k < 3; k++) x[k] = (f4 * z[k] - r[k]) * inv;
    x[3] = (dot3(w, f) - det * f4) * inv;
}

// Whether a row a x = b of the system is met to 1e-8 of the terms that cancel
// in it (not with a NaN or an infinity).  The step steers a search that ends
// by its own residual.  Of 300 random pairs each, a third of them with equal
// orientations, axes within 1:3, elimination for every step leaves 18 solves
// unconverged at blockiness 8 and 61 at 20, unchecked cofactors 20 and 68, and
// cofactors with this test 18 and 61; it sends 7 and 16 % of the steps to
// solve_pivoted there, and none at blockiness 4 or in random packings up to 8.
__device__ __forceinline__ bool row_met(const double *a, double b, const double *x)
{
    double left = -b, size = fabs(b);
    for (int j = 0; j < 4; j++) {
        left += a[j] * x[j];
        size += fabs(a[j] * x[j]);
    }
    return fabs(left) <= 1e-8 * size && size < INFINITY;
}

// The same system by Gauss-Jordan elimination with partial pivoting, lane ax
// of each four holding row ax (a, b); every lane receives x.  False when a
// pivot is zero.  All lanes of the warp take part.
__device__ __forceinline__ bool solve_pivoted(int lane, double *a, double b, double *x)
{
    const unsigned FULL = 0xffffffffu;
    const int ax = lane & 3;
    bool used = false, ok = true;
    double pivot = 1.0;
    int at[4];   // the row that each column was eliminated with
#pragma unroll
    for (int c = 0; c < 4; c++) {
        double v = used ? -1.0 : fabs(a[c]);
        int r = ax;
#pragma unroll
        for (int o = 1; o < 4; o <<= 1) {
            const double v2 = __shfl_xor_sync(FULL, v, o);
            const int r2 = __shfl_xor_sync(FULL, r, o);
            if (v2 > v || (v2 == v && r2 < r)) {
                v = v2;
                r = r2;
            }
        }
        ok = ok && v > 0.0;
        r = __shfl_sync(FULL, r, lane & 28);   // (NaNs compare false)
        at[c] = r;
        const int src = (lane & 28) + r;
        double p[4];
#pragma unroll
        for (int j = c; j < 4; j++) p[j] = __shfl_sync(FULL, a[j], src);
        const double pb = __shfl_sync(FULL, b, src);
        if (ax == r) {
            used = true;
            pivot = a[c];
        } else {
            const double m = a[c] / p[c];
#pragma unroll
            for (int j = c; j < 4; j++) a[j] -= m * p[j];
            b -= m * pb;
        }
    }
    const double q = b / pivot;
#pragma unroll
    for (int c = 0; c < 4; c++) x[c] = __shfl_sync(FULL, q, (lane & 28) + at[c]);
    return ok;
}

// The sum of a * b over the lanes of one body (4) or of the pair (8), the same
// bits in each of them.  Product and sums are rounded one by one: contracted,
// a lane would add its own unrounded product to its partner's rounded one, and
// the two lanes' sums would differ.
__device__ __forceinline__ double sum4(unsigned mask, double a, double b)
{
    double v = __dmul_rn(a, b);
    v = __dadd_rn(v, __shfl_xor_sync(mask, v, 1));
    return __dadd_rn(v, __shfl_xor_sync(mask, v, 2));
}
__device__ __forceinline__ double sum8(unsigned mask, double a, double b)
{
    const double v = sum4(mask, a, b);
    return __dadd_rn(v, __shfl_xor_sync(mask, v, 4));
}

// one lane's share of a body: its axis
struct Axis {
    double c[3], rc[3];      // body centre, the axis direction (a column of the rotation)
    double full, n_full;     // half-axis and blockiness of the particle
    double round;            // radius of the homotopy's starting sphere
    double s, inv, n, koef;  // of the current stage
    int ni;                  // integer exponent, or -1: the powers go through pow
};

// shape of stage fraction t (1: the particle itself); idle lanes keep inv = 0
__device__ __forceinline__ void axis_stage(Axis &X, bool idle, double t, bool last)
{
    X.s = last ? X.full : X.round + (X.full - X.round) * t;
    X.n = last ? X.n_full : 2.0 + (X.n_full - 2.0) * t;
    X.inv = idle ? 0.0 : 1.0 / X.s;
    X.koef = exp2(2.0 - X.n);   // 0.5^(n - 2)
    X.ni = comp_double(X.n, 2.0, 1e-2) || is_integer(X.n) ? (int)floor(X.n + 1e-2) : -1;
}

// The listed solves: first contacts (list 0; `guess`, when given, holds the
// network's output per item), then warm starts (list 1).  A group starts with
// the item of its own number and takes later ones from W.next.
__global__ void __launch_bounds__(128, 3) k_sq_solve(SqDev D, SqWork W, const int *__restrict__ own, int shearupdate,
                                                     const float4 *__restrict__ guess)
{
    const unsigned FULL = 0xffffffffu;
    const int lane = threadIdx.x & 31, gl = lane & 7, ax = gl & 3;
    const bool second = gl >= 4, idle = ax == 3;   // second: the lane's body is j
    const unsigned gmask = 0xffu << (lane & 24);
    const double tol1 = 1e-10, tol2 = 1e-12;
    const int nfirst = W.n[0], total = nfirst + W.n[1];
    const int ngroups = gridDim.x * (blockDim.x >> 3);
    int item = blockIdx.x * (blockDim.x >> 3) + (threadIdx.x >> 3);
    bool fresh = true;   // item is the group's own first one

    Axis X;
    int state = Q_IDLE, sl = 0, phase = 0, stage = 0, nstage = 0, maxit = kMaxNewton, used = 0;
    double ninv = 0.0, mid[3], size = 0.0;
    // the point evaluated next, and how its multiplier is found
    double p[3] = {0, 0, 0}, mut = 0.0;
    bool grad_mu = true;
    // the current iterate of the solve
    double pt[3], mu = 0.0, fi = 0.0, fj = 0.0, gA[3], gB[3], F[4], res1 = 0.0, merit1 = 0.0, dcur = 0.0;
    int it = 0;
    bool fail = false;
    // the Newton step, and the golden-section search along it
    double del[4] = {0, 0, 0, 0}, deltax = 0.0, ga = 0.0, gb = 1.0, resa = 0.0;
    // the line search of this lane's body
    double lx = 0.0, dl = 0.0, alpha = 0.0, amax = 0.0, f0 = 0.0, delta = 0.0;
    int lstate = 0, lit = 0, halv = 0;
    bool ldone = true;
    for (int k = 0; k < 3; k++) {
        X.c[k] = X.rc[k] = 0.0;
        mid[k] = pt[k] = gA[k] = gB[k] = F[k] = 0.0;
    }
    F[3] = 0.0;
    X.full = X.round = X.s = 1.0;
    X.n_full = X.n = 2.0;
    X.inv = 0.0;
    X.koef = 1.0;
    X.ni = 2;
    unsigned long long c_it = 0, c_sv = 0;
    unsigned c_pairs = 0, c_used = 0, c_rej = 0;

    for (;;) {
        if (state == Q_IDLE) {
            if (!fresh) {
                if (gl == 0) item = ngroups + atomicAdd(W.next, 1);
                item = __shfl_sync(gmask, item, lane & 24);
            }
            fresh = false;
            if (item >= total) {
                state = Q_DONE;
            } else {
                const bool first = item < nfirst;
                sl = first ? W.list[0][item] : W.list[1][item - nfirst];
                const int i = own[sl], j = D.nbr[sl];
                const dbl4 xi = D.x[i], xj = D.x[j], si = D.shape[i], sj = D.shape[j];
                const double ri = cbrt(si.x * si.y * si.z), rj = cbrt(sj.x * sj.y * sj.z);
                const double ratio = ri / (ri + rj);
                mid[0] = ratio * xj.x + (1.0 - ratio) * xi.x;
                mid[1] = ratio * xj.y + (1.0 - ratio) * xi.y;
                mid[2] = ratio * xj.z + (1.0 - ratio) * xi.z;
                const dbl4 q4 = D.q[second ? j : i], x4 = second ? xj : xi, s4 = second ? sj : si;
                const double q[4] = {q4.x, q4.y, q4.z, q4.w};
                double R[9];
                quat_to_mat(q, R);
                X.c[0] = x4.x;
                X.c[1] = x4.y;
                X.c[2] = x4.z;
                for (int k = 0; k < 3; k++)
                    X.rc[k] = idle ? 0.0 : (ax == 0 ? R[3 * k] : (ax == 1 ? R[3 * k + 1] : R[3 * k + 2]));
                X.full = idle ? 1e300 : (ax == 0 ? s4.x : (ax == 1 ? s4.y : s4.z));
                X.n_full = s4.w;
                X.round = idle ? 1e300 : (second ? rj : ri);
                const double nmax = fmax(si.w, sj.w);
                nstage = max((int)((nmax - 2.0) / 1.0 + 1), 10);
                ninv = 1.0 / (double)nstage;
                used = 0;
                stage = 0;
                it = 0;
                fail = false;
                grad_mu = true;
                maxit = kMaxNewton;
                c_pairs++;
                if (!first) {   // the previous point advanced with the mass-weighted contact-point velocity
                    phase = 2;
                    const dbl4 cp4 = D.cp[sl], wi4 = D.w[i], wj4 = D.w[j], vi4 = D.v[i], vj4 = D.v[j];
                    const double cp[3] = {cp4.x, cp4.y, cp4.z};
                    const double wi[3] = {wi4.x, wi4.y, wi4.z}, wj[3] = {wj4.x, wj4.y, wj4.z};
                    const double xci[3] = {cp[0] - xi.x, cp[1] - xi.y, cp[2] - xi.z};
                    const double xcj[3] = {cp[0] - xj.x, cp[1] - xj.y, cp[2] - xj.z};
                    double vri[3], vrj[3];
                    cross3(wi, xci, vri);
                    cross3(wj, xcj, vrj);
                    const double mi = vi4.w, mj = vj4.w;
                    const double vi[3] = {vi4.x, vi4.y, vi4.z}, vj[3] = {vj4.x, vj4.y, vj4.z};
                    for (int k = 0; k < 3; k++)
                        p[k] = cp[k] + ((vi[k] + vri[k]) * mi + (vj[k] + vrj[k]) * mj) / (mi + mj) * D.dt;
                } else if (guess) {   // the network's point (i's frame, over ri + rj) and multiplier
                    phase = 0;
                    const float4 g = guess[item];
                    const double s = ri + rj, pl[3] = {g.x * s, g.y * s, g.z * s};
                    const dbl4 qi4 = D.q[i];
                    const double qi[4] = {qi4.x, qi4.y, qi4.z, qi4.w};
                    double Ri[9];
                    quat_to_mat(qi, Ri);
                    matvec(Ri, pl, p);
                    p[0] += xi.x;
                    p[1] += xi.y;
                    p[2] += xi.z;
                    mut = (double)fabsf(g.w);
                    grad_mu = false;
                    maxit = kLearnedNewton;
                } else {
                    phase = 1;
                    for (int k = 0; k < 3; k++) p[k] = mid[k];
                }
                axis_stage(X, idle, 0.0, phase != 1);
                size = X.s;
                size = fmin(size, __shfl_xor_sync(gmask, size, 1));
                size = fmin(size, __shfl_xor_sync(gmask, size, 2));
                size = fmin(size, __shfl_xor_sync(gmask, size, 4));
                state = Q_INIT1;
            }
        }
        if (__all_sync(FULL, state == Q_DONE)) break;

        // ---- one evaluation for every group
        const bool line = state == Q_LINE;
        const double xl = line ? lx + delta * dl
                               : X.rc[0] * (p[0] - X.c[0]) + X.rc[1] * (p[1] - X.c[1]) + X.rc[2] * (p[2] - X.c[2]);
        const double u = xl * X.inv, au = fabs(u);
        const double p2 = X.ni >= 0 ? ipow(au, max(X.ni - 2, 0)) : pow_pos(au, X.n - 2.0);
        const double p1 = p2 * au;
        const double ka = X.koef * X.inv;
        const double g0 = ka * X.n * sgn(u) * p1;
        const double dnew = ka * (X.n * (X.n - 1.0) * p2) * X.inv;
        const double f_own = X.koef * (sum4(FULL, p1, au) - 1.0);
        double go[3];
        go[0] = sum4(FULL, line ? dl : X.rc[0], g0);
        go[1] = sum4(FULL, X.rc[1], g0);
        go[2] = sum4(FULL, X.rc[2], g0);
        double tA[3], tB[3];
        for (int k = 0; k < 3; k++) {
            const double gx = __shfl_xor_sync(FULL, go[k], 4);
            tA[k] = second ? gx : go[k];
            tB[k] = second ? go[k] : gx;
        }
        const double fx = __shfl_xor_sync(FULL, f_own, 4);
        const double tfi = second ? fx : f_own, tfj = second ? f_own : fx;

        // ---- what it means for the group's solve (calc_F of the trial point)
        bool step = false, end = false;
        if (state != Q_LINE && state != Q_DONE) {
            const double aa = dot3(tA, tA), bb = dot3(tB, tB);
            double mu_sq, muo;
            if (grad_mu) {
                mu_sq = -dot3(tA, tB) / bb;
                muo = sqrt(fabs(mu_sq));
            } else {
                mu_sq = mut * mut;
                muo = mut;
            }
            const double G[4] = {tA[0] + mu_sq * tB[0], tA[1] + mu_sq * tB[1], tA[2] + mu_sq * tB[2], tfi - tfj};
            double v[3];
            cross3(tA, tB, v);
            const double sine = fabs(dot3(v, v) / (aa * bb));
            const double aaa = fabs(G[3]) / (fmax(fabs(tfi), fabs(tfj)) + 1e-16);
            const double merit = fmax(sine, aaa * aaa);
            const double res = G[0] * G[0] + G[1] * G[1] + G[2] * G[2] + G[3] * G[3];
            bool take = false, accept = false, converged = false;
            switch (state) {
            case Q_INIT1:
                take = true;
                if (merit < tol1) {
                    end = true;
                } else {   // the start to compare with: the sphere solution
                    grad_mu = true;
                }
                break;
            case Q_INIT2:
                take = !(res1 < res);
                break;
            case Q_TRIAL:
                if (res < res1 || merit < tol1 || deltax < tol2 * size) {
                    take = accept = true;
                    converged = merit < tol1 || deltax < tol2 * size;
                } else {
                    ga = 0.0;
                    gb = 1.0;
                    state = Q_GOLD_A;
                }
                break;
            case Q_GOLD_A:
                resa = res;
                state = Q_GOLD_B;
                break;
            case Q_GOLD_B:
                if (fmin(resa, res) < res1) {
                    if (resa < res) {
                        state = Q_GOLD_TAKE;   // evaluated again, to be taken
                    } else {
                        take = accept = true;
                        converged = merit < tol1;
                    }
                } else {
                    const double al1 = gb - (gb - ga) * kPhiInv, al2 = ga + (gb - ga) * kPhiInv;
                    if (resa > res) ga = al1;
                    else gb = al2;
                    if (fabs(gb - ga) > 1e-8) {
                        state = Q_GOLD_A;
                    } else {
                        take = accept = true;
                        converged = merit < tol1;
                    }
                }
                break;
            default:   // Q_GOLD_TAKE
                take = accept = true;
                converged = merit < tol1;
            }
            const double before = res1;
            if (take) {
                for (int k = 0; k < 3; k++) {
                    pt[k] = p[k];
                    gA[k] = tA[k];
                    gB[k] = tB[k];
                }
                for (int k = 0; k < 4; k++) F[k] = G[k];
                mu = muo;
                fi = tfi;
                fj = tfj;
                dcur = dnew;
                res1 = res;
                merit1 = merit;
            }
            if (accept) {
                if (fabs(before - res1) < 1e-3 * fmax(before, res1)) converged = true;
                if (it >= maxit) fail = true;
                if (converged || fail) end = true;
                else step = true;
            } else if (state == Q_INIT2) {
                if (merit1 < tol1) end = true;
                else step = true;
            } else if (state == Q_INIT1 && !end) {
                for (int k = 0; k < 3; k++) p[k] = mid[k];
                state = Q_INIT2;
            } else if (state >= Q_GOLD_A && state <= Q_GOLD_TAKE) {
                const double al = state == Q_GOLD_B ? ga + (gb - ga) * kPhiInv : gb - (gb - ga) * kPhiInv;
                for (int k = 0; k < 3; k++) p[k] = pt[k] - al * del[k];
                mut = mu - al * del[3];
            }
        }
        __syncwarp();

        // ---- Newton steps (all lanes take part in the sums; the groups that asked use the result)
        if (__any_sync(FULL, step)) {
            const double w = second ? mu * mu * dcur : dcur;
            const double r0 = X.rc[0] * w, r1 = X.rc[1] * w, r2 = X.rc[2] * w;
            double h[6], cc[3], dd[3];
            h[0] = sum8(FULL, r0, X.rc[0]);
            h[1] = sum8(FULL, r0, X.rc[1]);
            h[2] = sum8(FULL, r0, X.rc[2]);
            h[3] = sum8(FULL, r1, X.rc[1]);
            h[4] = sum8(FULL, r1, X.rc[2]);
            h[5] = sum8(FULL, r2, X.rc[2]);
            for (int k = 0; k < 3; k++) {
                cc[k] = 2.0 * mu * gB[k];
                dd[k] = gA[k] - gB[k];
            }
            double x[4];
            solve_bordered(h, cc, dd, F, F[3], x);
            // each lane looks at one row, lanes 3 and 7 at the border's
            double row[4];
            row[0] = idle ? dd[0] : (ax == 0 ? h[0] : (ax == 1 ? h[1] : h[2]));
            row[1] = idle ? dd[1] : (ax == 0 ? h[1] : (ax == 1 ? h[3] : h[4]));
            row[2] = idle ? dd[2] : (ax == 0 ? h[2] : (ax == 1 ? h[4] : h[5]));
            row[3] = idle ? 0.0 : (ax == 0 ? cc[0] : (ax == 1 ? cc[1] : cc[2]));
            const double rhs = idle ? F[3] : (ax == 0 ? F[0] : (ax == 1 ? F[1] : F[2]));
            const unsigned poor = __ballot_sync(FULL, step && !row_met(row, rhs, x));
            bool ok = true;
            if (poor) {
                double y[4];
                const bool solved = solve_pivoted(lane, row, rhs, y);
                if (poor & gmask) {
                    ok = solved;
                    for (int k = 0; k < 4; k++) x[k] = y[k];
                }
            }
            for (int k = 0; k < 4; k++) ok = ok && !isnan(x[k]);
            if (step) {
                it++;
                if (!ok) {
                    fail = true;
                    end = true;
                } else {
                    deltax = fmax(fmax(fabs(x[0]), fabs(x[1])), fabs(x[2]));
                    if (deltax == 0.0) {
                        if (it >= maxit) fail = true;
                        end = true;
                    } else {
                        for (int k = 0; k < 4; k++) del[k] = x[k];
                        for (int k = 0; k < 3; k++) p[k] = pt[k] - del[k];
                        mut = mu - del[3];
                        grad_mu = false;
                        state = Q_TRIAL;
                    }
                }
            }
        }

        // the first lane's decision for the group
        const int decided = __shfl_sync(FULL, state | (end ? 16 : 0), lane & 24);
        state = decided & 15;
        end = (decided & 16) != 0;

        // ---- the end of one solve: the next stage, the homotopy after a
        // rejected guess, or the item's result
        if (end) {
            c_it += it;
            c_sv++;
            it = 0;
            const unsigned verdict =
                __shfl_sync(gmask, (phase == 0 && (fail || !(merit1 < 1e-10)) ? 1u : 0u) |
                                       (fmax(fi, fj) < 0.0 ? 2u : 0u), lane & 24);
            const bool rejected = verdict & 1u, overlap = verdict & 2u;
            fail = false;
            if (rejected || (phase == 1 && stage < nstage)) {
                if (rejected) {
                    phase = 1;
                    used = -1;
                    stage = 0;
                    maxit = kMaxNewton;
                    for (int k = 0; k < 3; k++) p[k] = mid[k];
                } else {
                    stage++;
                    for (int k = 0; k < 3; k++) p[k] = pt[k];
                }
                axis_stage(X, idle, (double)stage * ninv, false);
                size = X.s;
                size = fmin(size, __shfl_xor_sync(gmask, size, 1));
                size = fmin(size, __shfl_xor_sync(gmask, size, 2));
                size = fmin(size, __shfl_xor_sync(gmask, size, 4));
                grad_mu = true;
                state = Q_INIT1;
            } else {
                if (phase == 0) used = 1;
                if (used == 1) c_used++;
                if (used == -1) c_rej++;
                if (gl == 0) D.cp[sl] = dbl4{pt[0], pt[1], pt[2], 0.0};
                if (!overlap) {
                    if (gl == 0) D.state[sl] = CLOSE;
                    state = Q_IDLE;
                } else {   // the overlap along the normal: a line search per body
                    axis_stage(X, idle, 1.0, true);
                    double en[3] = {gB[0] - gA[0], gB[1] - gA[1], gB[2] - gA[2]};
                    const double nrm = sqrt(dot3(en, en));
                    const double ninv2 = nrm == 0. ? 0. : 1. / nrm;
                    for (int k = 0; k < 3; k++) {
                        en[k] *= ninv2;
                        gA[k] = en[k];   // kept for the forces
                        if (!second) en[k] = -en[k];
                    }
                    const double t[3] = {pt[0] - X.c[0], pt[1] - X.c[1], pt[2] - X.c[2]};
                    lx = dot3(X.rc, t);
                    dl = dot3(X.rc, en);
                    const double2 al = D.alpha[sl];
                    alpha = second ? al.y : al.x;
                    delta = 0.0;
                    lstate = lit = halv = 0;
                    double smin = X.s;
                    smin = fmin(smin, __shfl_xor_sync(gmask, smin, 1));
                    smin = fmin(smin, __shfl_xor_sync(gmask, smin, 2));
                    const double x0 = lx * X.inv, nx = dl * X.inv;
                    const double qa = sum4(gmask, nx, nx), qb = 2.0 * sum4(gmask, x0, nx);
                    const double qc = sum4(gmask, x0, x0) - 1.0;
                    ldone = false;
                    if (comp_double(X.n, 2.0, 1e-2)) {   // an ellipsoid: the quadratic
                        const double eps0 = 1e-14;
                        const double disc = qb * qb - 4.0 * qa * qc, tai = 0.5 / qa;
                        double a1, a2;
                        if (disc < 0) {
                            a1 = -qb * tai;
                            a2 = a1;
                        } else {
                            const double sD = sqrt(disc);
                            a1 = (-qb + sD) * tai;
                            a2 = (-qb - sD) * tai;
                        }
                        if (a1 > -eps0 && a2 < -eps0) alpha = a1;
                        else if (a1 < -eps0 && a2 > -eps0) alpha = a2;
                        else if (a1 < -eps0 && a2 < -eps0) alpha = fmax(a1, a2);
                        else alpha = fmin(a1, a2);
                        ldone = true;
                    } else {
                        amax = 0.5 * smin / sqrt(dot3(en, en));
                        alpha = alpha < -amax ? -amax : (alpha > amax ? amax : alpha);
                        lx += alpha * dl;
                    }
                    state = Q_LINE;
                }
            }
        } else if (line) {
            // ---- the line search (Superquadric::surface_line_intersection, src/superquadric.cpp:712-818,
            // 20 iterations, halvings; extended overlap src/math_extra_liggghts_superquadric.cpp:1489)
            const double eps = 1e-16, f = f_own, fder = go[0];
            if (!ldone) {
                bool top = false, have = false;
                double fd = fder;
                if (lstate == 0) {
                    f0 = f;
                    if (fabs(f0) < eps) ldone = true;
                    else top = true;
                } else if (lstate == 1) {
                    if (fabs(f) < fabs(f0) || fabs(f) < eps * X.koef) {
                        f0 = f;
                        alpha += delta;
                        lx += delta * dl;
                        if (++lit >= 20) ldone = true;
                        else top = true;
                    } else {   // a step that no halving improves would only repeat itself
                        delta *= 0.5;
                        if (!(fabs(delta) > eps && ++halv < 80)) ldone = true;
                    }
                } else {
                    delta = fder < 0.0 ? -1e-10 : 1e-10;
                    have = true;
                }
                if (top) {
                    if (fabs(f0) < eps * X.koef) {
                        ldone = true;
                    } else if (fabs(fd) < 1e-10) {
                        delta = 1e-10;
                        lstate = 2;
                    } else {
                        delta = -f0 / fd;
                        delta = delta < -amax ? -amax : (delta > amax ? amax : delta);
                        have = true;
                    }
                }
                if (have) {
                    if (fabs(delta) <= eps) {
                        alpha += delta;
                        ldone = true;
                    } else {
                        halv = 0;
                        lstate = 1;
                    }
                }
            }
        }
        __syncwarp();

        // ---- both lines done: contact forces (non-spherical kinematics, Hertz, tangential history)
        ldone = __shfl_sync(FULL, (int)ldone, lane & 28) != 0;   // each body's first lane decides for it
        const bool both = __shfl_xor_sync(FULL, (int)ldone, 4) != 0 && ldone;
        const double aother = __shfl_xor_sync(FULL, alpha, 4);
        if (state == Q_LINE && both) {
            const double al_x = second ? aother : alpha, al_y = second ? alpha : aother;
            const double deltan = fabs(al_x) + fabs(al_y);
            const double en[3] = {gA[0], gA[1], gA[2]};
            const int i = own[sl], j = D.nbr[sl];
            const dbl4 xi4 = D.x[i], xj4 = D.x[j];
            const dbl4 vi4 = D.v[i], vj4 = D.v[j], wi4 = D.w[i], wj4 = D.w[j], ii4 = D.inert[i], ij4 = D.inert[j];
            const double wi[3] = {wi4.x, wi4.y, wi4.z}, wj[3] = {wj4.x, wj4.y, wj4.z};
            const double xci[3] = {pt[0] - xi4.x, pt[1] - xi4.y, pt[2] - xi4.z};
            const double xcj[3] = {pt[0] - xj4.x, pt[1] - xj4.y, pt[2] - xj4.z};
            double vri[3], vrj[3], vrel[3];
            cross3(wi, xci, vri);
            cross3(wj, xcj, vrj);
            const double vi[3] = {vi4.x, vi4.y, vi4.z}, vj[3] = {vj4.x, vj4.y, vj4.z};
            for (int k = 0; k < 3; k++) vrel[k] = vi[k] - vj[k] + (vri[k] - vrj[k]);
            const double vn = dot3(vrel, en);
            const double vtr[3] = {vrel[0] - vn * en[0], vrel[1] - vn * en[1], vrel[2] - vn * en[2]};
            const double radi = ii4.w, radj = ij4.w, mi = vi4.w, mj = vj4.w, meff = mi * mj / (mi + mj);
            const double reff = radi * radj / (radi + radj);
            const double sqrtval = sqrt(reff * deltan);
            const double Sn = 2. * D.Yeff * sqrtval, St = 8. * D.Geff * sqrtval;
            const double kn = 4. / 3. * D.Yeff * sqrtval, kt = St;
            const double c56 = 0.91287092917527685576161630466800355658790782499663875;
            const double gamman = -2. * c56 * D.betaeff * sqrt(Sn * meff);
            const double gammat = -2. * c56 * D.betaeff * sqrt(St * meff);
            const double Fn = -gamman * vn + kn * deltan;
            const double Fi[3] = {Fn * en[0], Fn * en[1], Fn * en[2]}, Fnj[3] = {-Fi[0], -Fi[1], -Fi[2]};
            double Ti[3], Tj[3];
            cross3(xci, Fi, Ti);
            cross3(xcj, Fnj, Tj);
            const dbl4 sh4 = D.shear[sl];
            double sh[3] = {sh4.x, sh4.y, sh4.z};
            if (shearupdate) {
                for (int k = 0; k < 3; k++) sh[k] += vtr[k] * D.dt;
                const double rsht = dot3(sh, en);
                for (int k = 0; k < 3; k++) sh[k] -= rsht * en[k];
            }
            const double shrmag = sqrt(dot3(sh, sh));
            double Ft[3] = {-(kt * sh[0]), -(kt * sh[1]), -(kt * sh[2])};
            const double Ft_shear = kt * shrmag, Ft_friction = D.mu * fabs(Fn);
            if (Ft_shear > Ft_friction) {
                if (shrmag != 0.0) {
                    const double ratio = Ft_friction / Ft_shear;
                    for (int k = 0; k < 3; k++) Ft[k] *= ratio;
                    if (shearupdate)
                        for (int k = 0; k < 3; k++) sh[k] = -Ft[k] / kt;
                } else {
                    Ft[0] = Ft[1] = Ft[2] = 0.0;
                }
            } else {
                for (int k = 0; k < 3; k++) Ft[k] -= gammat * vtr[k];
            }
            double tti[3], ttj[3];
            const double Ftj[3] = {-Ft[0], -Ft[1], -Ft[2]};
            cross3(xci, Ft, tti);
            cross3(xcj, Ftj, ttj);
            __syncwarp(gmask);   // every lane has read the slot's shear
            if (gl == 0) {
                D.alpha[sl] = make_double2(al_x, al_y);
                D.shear[sl] = dbl4{sh[0], sh[1], sh[2], 0.0};
                D.pfi[sl] = dbl4{Fi[0] + Ft[0], Fi[1] + Ft[1], Fi[2] + Ft[2], 1.0};
                D.pti[sl] = dbl4{Ti[0] + tti[0], Ti[1] + tti[1], Ti[2] + tti[2], 0.0};
                D.ptj[sl] = dbl4{Tj[0] + ttj[0], Tj[1] + ttj[1], Tj[2] + ttj[2], 0.0};
                D.flag[sl] |= 5;
                D.state[sl] = INTERSECT;
            }
            state = Q_IDLE;
        }
        __syncwarp();
    }
    if (gl == 0 && c_pairs) {
        atomicAdd(&D.cnt[0], c_it);
        atomicAdd(&D.cnt[1], c_sv);
        atomicAdd(&D.cnt[2], (unsigned long long)c_pairs);
        if (c_used) atomicAdd(&D.cnt[3], (unsigned long long)c_used);
        if (c_rej) atomicAdd(&D.cnt[4], (unsigned long long)c_rej);
    }
}

// The learned guesses of the first contacts, 32 pairs per warp on the tensor
// cores; guess[q] is the network's output for item q of list 0.
__global__ void __launch_bounds__(128) k_sq_guess(SqDev D, SqWork W, const int *__restrict__ own,
                                                  float4 *__restrict__ guess)
{
    __shared__ __align__(16) MlpInfer S;
    const int n = W.n[0];
    if ((int)(blockIdx.x * blockDim.x) >= n) return;
    mlp_stage(S, D.mlp);
    __syncthreads();
    const int lane = threadIdx.x & 31;
    for (int base = blockIdx.x * blockDim.x + (threadIdx.x & ~31); base < n; base += gridDim.x * blockDim.x) {
        const int q = base + lane;
        float feat[kMlpIn], out[kMlpOut];
        if (q < n) {
            const int sl = W.list[0][q], i = own[sl], j = D.nbr[sl];
            const dbl4 xi4 = D.x[i], xj4 = D.x[j], qi4 = D.q[i], qj4 = D.q[j], si4 = D.shape[i], sj4 = D.shape[j];
            const double ci[3] = {xi4.x, xi4.y, xi4.z}, cj[3] = {xj4.x, xj4.y, xj4.z};
            const double qi[4] = {qi4.x, qi4.y, qi4.z, qi4.w}, qj[4] = {qj4.x, qj4.y, qj4.z, qj4.w};
            const double si[3] = {si4.x, si4.y, si4.z}, sj[3] = {sj4.x, sj4.y, sj4.z};
            pair_features_of(ci, qi, si, si4.w, cj, qj, sj, sj4.w, feat);
        }
        mlp_infer_warp(S, q < n, feat, out);
        if (q < n) guess[q] = make_float4(out[0], out[1], out[2], out[3]);
    }
}

}  // namespace sq
}  // namespace gb2
