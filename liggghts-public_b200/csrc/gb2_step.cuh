// gb2_step.cuh -- the fused pair-step kernel (one full time step per owned
// atom).  Instantiated with SPLIT=false by the bit-exact FP64 unit and with
// SPLIT=true by the split-precision unit (gb2_split.cu).
#pragma once

#include <type_traits>

#include "gb2_device.cuh"

namespace gb2 {
// Programmatic dependent launch: the pair step lets the tail kernel be
// scheduled as soon as all of its blocks are running; the tail kernel does
// what does not need the pair sums first and then waits for the pair step
// to complete (all its memory operations visible).  The next step's pair step
// is the tail kernel's dependent in turn: it may start early, but lets its own
// tail kernel start only after it has waited, so a tail kernel never runs
// beside the previous step's.
__device__ __forceinline__ void grid_dep_launch() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void grid_dep_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

__device__ __forceinline__ void prefetch_l1(const void *p) { asm volatile("prefetch.global.L1 [%0];" ::"l"(p)); }

// A kernel of a step queued ahead returns at once when an earlier step has
// asked for a neighbour rebuild (that step's successors are redone after it).
__device__ __forceinline__ bool step_cancelled(const Dev &D) { return D.dstop && *(volatile int *)D.dstop < D.step; }

// Atoms per warp of the tail kernel: lanes 0..kTailAtoms-1 own one atom
// each, all 32 lanes share the evaluation of their mesh candidates.
#ifndef GB2_TAIL_ATOMS
#define GB2_TAIL_ATOMS 8
#endif
constexpr int kTailAtoms = GB2_TAIL_ATOMS;

// One touching pair of the warp-compacted evaluation: owner kk, the other
// atom, the half-list slot s of the pair (in kk's list when own, in other's
// list otherwise).  A j-side entry is evaluated from kk's side with the
// shear negated; an own entry updates kk's shear slot in the write buffer
// and sets the contact flag.  res receives the pair's force and torque on kk.
// EARLY: called before the kernel's wait, so the records come from L2.
template <bool ROLLING, bool SPLIT, bool ONE, bool EARLY = false, typename Real>
__device__ __forceinline__ void eval_item(const Dev &D, int kk, int other, int s, bool own, bool upd, Real *res)
{
    const int cap = D.cap;
    const int e = s * cap + kk;
    const double sgn = own ? 1.0 : -1.0;
    const int hrow = own ? kk : other;
    const auto ld = [](const dbl4 *p) { return EARLY ? ldrec_l2(p) : ldrec(p); };
    const dbl4 pkk = ld(&D.pos[kk]);
    const dbl4 po = ld(&D.pos[other]);
    const double delx = pkk.x - po.x;
    const double dely = pkk.y - po.y;
    const double delz = pkk.z - po.z;
    const double rsq = delx * delx + dely * dely + delz * delz;
    // material lookup in the reference's (owner, neighbour) order
    const MatPair &M = ONE ? D.mat1 : (own ? mat(D, D.type[kk], D.type[other]) : mat(D, D.type[other], D.type[kk]));
    if constexpr (SPLIT) {
        const flt8 a = ldkin(&D.kin[kk]), b = ldkin(&D.kin[other]);
        const double r = sqrt(rsq);
        const double deltan = (pkk.w + po.w) - r;   // FP64 overlap
        const float va[3] = {a.vx, a.vy, a.vz}, wa[3] = {a.wx, a.wy, a.wz};
        const float vb[3] = {b.vx, b.vy, b.vz}, wb[3] = {b.wx, b.wy, b.wz};
        const float fs = (float)sgn;
        const dbl4 h = ld(&D.hist[s * cap + hrow]);
        float sh[3] = {fs * (float)h.x, fs * (float)h.y, fs * (float)h.z};
        ContactOutF o;
        pair_contact_f32(M, (float)delx, (float)dely, (float)delz, (float)r, (float)deltan, (float)pkk.w,
                         (float)po.w, va, vb, wa, wb, a.m, b.m, sh, upd, (float)D.dt, ROLLING, D.tdamp != 0, o);
        if (own && upd) D.hist_out[e] = dbl4{(double)sh[0], (double)sh[1], (double)sh[2], 0.0};
        for (int c = 0; c < 3; c++) {
            res[c] = o.F[c];
            res[3 + c] = o.T[c];
        }
    } else {
        const dbl4 vk4 = ld(&D.vel[kk]), wk4 = ld(&D.omg[kk]);
        const dbl4 vo4 = ld(&D.vel[other]), wo4 = ld(&D.omg[other]);
        const double vk[3] = {vk4.x, vk4.y, vk4.z}, wk[3] = {wk4.x, wk4.y, wk4.z};
        const double vo[3] = {vo4.x, vo4.y, vo4.z}, wo[3] = {wo4.x, wo4.y, wo4.z};
        const dbl4 h = ld(&D.hist[s * cap + hrow]);
        double sh[3] = {sgn * h.x, sgn * h.y, sgn * h.z};   // exact: multiplying by +-1 only flips the sign
        ContactOut o;
        if (!pair_contact_fast(M, delx, dely, delz, rsq, pkk.w, po.w, vk, vo, wk, wo, vk4.w, vo4.w, sh, upd, D.dt,
                               ROLLING, D.tdamp != 0, o)) {
            // an operand outside the fast arithmetic's range: read again, so that
            // this rare path keeps nothing alive through the other
            const auto again = [](const dbl4 *p) { return EARLY ? ldrec_l2(p) : *p; };
            const dbl4 p1 = again(&D.pos[kk]), p2 = again(&D.pos[other]), v1 = again(&D.vel[kk]),
                       v2 = again(&D.vel[other]), w1 = again(&D.omg[kk]), w2 = again(&D.omg[other]),
                       h1 = again(&D.hist[s * cap + hrow]);
            const auto type_again = [&D](int a) { return *(const volatile int *)&D.type[a]; };
            const double dx = p1.x - p2.x, dy = p1.y - p2.y, dz = p1.z - p2.z;
            const double va[3] = {v1.x, v1.y, v1.z}, vb[3] = {v2.x, v2.y, v2.z};
            const double wa[3] = {w1.x, w1.y, w1.z}, wb[3] = {w2.x, w2.y, w2.z};
            sh[0] = sgn * h1.x;
            sh[1] = sgn * h1.y;
            sh[2] = sgn * h1.z;
            const MatPair &M1 = ONE ? D.mat1 : mat(D, type_again(own ? kk : other), type_again(own ? other : kk));
            pair_contact<false>(M1, dx, dy, dz, dx * dx + dy * dy + dz * dz, p1.w, p2.w, va, vb, wa, wb, v1.w, v2.w, sh,
                                upd, D.dt, ROLLING, D.tdamp != 0, o);
        }
        if (own && upd) D.hist_out[e] = dbl4{(double)sh[0], (double)sh[1], (double)sh[2], 0.0};
        for (int c = 0; c < 3; c++) {
            res[c] = o.F[c];
            res[3 + c] = o.T[c];
        }
    }
}

// The pair sums of an atom k with more than 64 reverse or own entries, by a
// whole warp: the entries of a side are screened 128 at a time, the touching
// ones listed in order (list: kLongList ints of the warp's shared memory),
// evaluated one per lane, and added in list order -- the reference's order --
// by every lane.  What bounds it is the chain of dependent gathers, so the
// entries of four chunks are in flight together; one lane taking the entries
// one by one (a 3 mm sphere in a bed of 0.3 mm spheres has hundreds) set the
// whole step's time.  Out of line, as inlined it would take part in the tail
// kernel's register allocation (the call costs spills as well, see k_pair_tail).
// FP64 in both precisions, records from L2 (called before the wait).
constexpr int kLongList = kTailAtoms * 64;

template <bool ROLLING>
__device__ __noinline__ void long_atom(const Dev &D, int k, int nr, int nn, bool upd, int *list, ContactOut &acc)
{
    const unsigned FULL = 0xffffffffu;
    const int cap = D.cap, lane = threadIdx.x & 31;
    const dbl4 pk = ldrec_l2(&D.pos[k]);
    for (int c = 0; c < 3; c++) acc.F[c] = acc.T[c] = 0.0;
    for (int side = 0; side < 2; side++) {
        const int tot = side ? nn : nr;
        const int *idx = side ? D.nbr : D.rev;
        int n = 0;
        for (int base = 0; base < tot; base += 128) {
            int j[4];
            dbl4 q[4];
#pragma unroll
            for (int u = 0; u < 4; u++) {
                const int e = base + 32 * u + lane;
                j[u] = e < tot ? ld_stream(&idx[e * cap + k]) : k;
            }
#pragma unroll
            for (int u = 0; u < 4; u++) q[u] = ldrec_l2(&D.pos[j[u]]);
#pragma unroll
            for (int u = 0; u < 4; u++) {
                const int e = base + 32 * u + lane;
                const bool t = e < tot && touching(pk, q[u]);
                if (side && upd && e < tot && !t) D.hist_out[e * cap + k] = ldrec_l2(&D.hist[e * cap + k]);
                const unsigned m = __ballot_sync(FULL, t);
                if (t) list[n + __popc(m & ((1u << lane) - 1u))] = e;
                n += __popc(m);
            }
            __syncwarp();
            if (n > kLongList - 128 || base + 128 >= tot) {
                for (int b = 0; b < n; b += 32) {
                    double res[6] = {0., 0., 0., 0., 0., 0.};
                    if (b + lane < n) {
                        const int e = list[b + lane];
                        const int s = side ? e : (int)D.revs[e * cap + k];
                        if (side)   // CONTACT_NORMAL_MODEL | CONTACT_TANGENTIAL_MODEL
                            D.flag[e * cap + k] = __ldcg(&D.flag[e * cap + k]) | 5;
                        eval_item<ROLLING, false, false, true>(D, k, __ldg(&idx[e * cap + k]), s, side == 1, upd, res);
                    }
                    const int cnt = min(32, n - b);
                    for (int t = 0; t < cnt; t++)
#pragma unroll
                        for (int c = 0; c < 3; c++) {
                            acc.F[c] += __shfl_sync(FULL, res[c], t);
                            acc.T[c] += __shfl_sync(FULL, res[3 + c], t);
                        }
                }
                n = 0;
                __syncwarp();
            }
        }
    }
}

// FP64: plain in-order sum.  Split: FP32 sum with Kahan compensation kc.
// v: the item's column of the staged results (components 32 apart).
template <bool SPLIT, typename Real>
__device__ __forceinline__ void sum_item(Real *as, Real *kc, const Real *v)
{
#pragma unroll
    for (int c = 0; c < 6; c++) {
        if constexpr (SPLIT) {
            const float y = v[32 * c] - kc[c];
            const float t = as[c] + y;
            kc[c] = (t - as[c]) - y;
            as[c] = t;
        } else {
            as[c] += v[32 * c];
        }
    }
}

template <bool SPLIT, typename Real>
__device__ __forceinline__ void pair_total(const Real *as, const Real *kc, ContactOut &acc)
{
#pragma unroll
    for (int c = 0; c < 3; c++) {
        if constexpr (SPLIT) {
            acc.F[c] = (double)as[c] - (double)kc[c];
            acc.T[c] = (double)as[3 + c] - (double)kc[3 + c];
        } else {
            acc.F[c] = as[c];
            acc.T[c] = as[3 + c];
        }
    }
}

// store_f / FixNVESphere::final_integrate / the next step's initial_integrate
// with the displacement test, for one atom whose total force is in acc
// FixInsertStream::end_of_step (src/fix_insert_stream.cpp:868-935) for atom
// i: a particle the stream inserted and has not released moves with its
// integration velocity from its insertion position (x = x_ins + v_int
// (step - i_step) dt, v = v_int, omega = 0); at its release step it gets the
// release velocity and omega.  Returns true when it applies; the atom's
// force and torque then read zero.
__device__ __forceinline__ bool stream_hold(const Dev &D, int i, dbl4 &x, dbl4 &v, dbl4 &w)
{
    const dbl4 r0 = D.rel[i];
    if (r0.w < 1e-13 && r0.w > -1e-13) return false;   // never inserted by the stream
    const dbl4 r1 = D.rel[D.cap + i];
    const int i_step = static_cast<int>(r0.w + 1e-14);
    const int r_step = static_cast<int>(r1.w + 1e-14);
    if (D.step > r_step) return false;
    const double time_elapsed = (D.step - i_step) * D.dt;
    x.x = r0.x + r1.x * time_elapsed;
    x.y = r0.y + r1.y * time_elapsed;
    x.z = r0.z + r1.z * time_elapsed;
    if (D.step == r_step) {
        const dbl4 r2 = D.rel[2 * D.cap + i], r3 = D.rel[3 * D.cap + i];
        v.x = r2.x, v.y = r2.y, v.z = r2.z;
        w.x = r3.x, w.y = r3.y, w.z = r3.z;
    } else {
        v.x = r1.x, v.y = r1.y, v.z = r1.z;
        w.x = 0.0, w.y = 0.0, w.z = 0.0;
    }
    return true;
}

template <bool SPLIT>
__device__ __forceinline__ void atom_store_integrate(const Dev &D, int i, const dbl4 &pi, dbl4 vi4, dbl4 wi4,
                                                     const dbl4 &hold, int integrate, int fuse_next, int store_f,
                                                     const ContactOut &acc_in)
{
    // an atom held by fix insert/stream ends the step where end_of_step puts
    // it, with zero force and torque (the next initial_integrate reads them)
    ContactOut acc = acc_in;
    dbl4 pcur = pi;
    if (D.rel && integrate && stream_hold(D, i, pcur, vi4, wi4)) {
        for (int c = 0; c < 3; c++) acc.F[c] = acc.T[c] = 0.0;
        integrate = 2;   // final_integrate's result is replaced
    }
    if (store_f) {
        dbl4 Fo, To;
        Fo.x = acc.F[0];
        Fo.y = acc.F[1];
        Fo.z = acc.F[2];
        Fo.w = 0.0;
        To.x = acc.T[0];
        To.y = acc.T[1];
        To.z = acc.T[2];
        To.w = 0.0;
        D.f[i] = Fo;
        D.tq[i] = To;
    }
    if (integrate) {
        // FixNVESphere::final_integrate (src/fix_nve_sphere.cpp:208-246)
        const double dtf = 0.5 * D.dt * 1.0;
        const double dtfrotate = dtf / 0.4;
        const double dtfm = dtf / (vi4.w * 1.0);
        const double dtirotate = dtfrotate / (pi.w * pi.w * vi4.w);
        if (integrate == 1) {
            vi4.x += dtfm * acc.F[0];
            vi4.y += dtfm * acc.F[1];
            vi4.z += dtfm * acc.F[2];
            wi4.x += dtirotate * acc.T[0];
            wi4.y += dtirotate * acc.T[1];
            wi4.z += dtirotate * acc.T[2];
        }
        if (fuse_next) {
            // next step's FixNVESphere::initial_integrate with the same force,
            // then Neighbor::check_distance's displacement test
            const double dtv = D.dt;
            vi4.x += dtfm * acc.F[0];
            vi4.y += dtfm * acc.F[1];
            vi4.z += dtfm * acc.F[2];
            dbl4 p = pcur;
            p.x += dtv * vi4.x;
            p.y += dtv * vi4.y;
            p.z += dtv * vi4.z;
            wi4.x += dtirotate * acc.T[0];
            wi4.y += dtirotate * acc.T[1];
            wi4.z += dtirotate * acc.T[2];
            D.pos_out[i] = p;
            const dbl4 h = hold;
            const double delx = p.x - h.x, dely = p.y - h.y, delz = p.z - h.z;
            if (delx * delx + dely * dely + delz * delz > D.triggersq) {
                *D.dflag = 1;
                if (D.dstop) {
                    atomicMin(D.dstop, D.step);
                    *(volatile int *)D.hstop = 1;
                }
            }
            // the next step's forward communication: the atom's periodic
            // images move with it (its own kernel, which copied every ghost
            // record again, took 4-5 us of each step)
            if (D.ghead)
                for (int g = D.ghead[i]; g >= 0; g = D.gnext[g]) {
                    const dbl4 s = D.gshift[g];
                    const int gi = D.nlocal + g;
                    D.pos_out[gi] = dbl4{p.x + s.x, p.y + s.y, p.z + s.z, p.w};
                    D.vel_out[gi] = vi4;
                    D.omg_out[gi] = wi4;
                    if constexpr (SPLIT) D.kin_out[gi] = make_kin(vi4, wi4);
                }
        }
        D.vel_out[i] = vi4;
        D.omg_out[i] = wi4;
        if constexpr (SPLIT) D.kin_out[i] = make_kin(vi4, wi4);
    }
}

// The last step of a run (no fused initial_integrate): positions of the atoms
// fix insert/stream holds, set in place once the step's kernels are done.
static __global__ void k_stream_positions(Dev D)
{
    if (step_cancelled(D)) return;   // D.pos is then an earlier step's
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= D.nlocal) return;
    dbl4 x = D.pos[i], v, w;
    if (stream_hold(D, i, x, v, w)) D.pos[i] = x;
}

// Own slots that touch and did not in the previous step (prevm; empty after
// a build and in setup) get their contact flag; shear of own slots that
// stopped touching is carried into the write buffer, and the touching mask is
// kept for the next step.
__device__ __forceinline__ void atom_hist_tail(const Dev &D, int k, unsigned long long prevm,
                                               unsigned long long mown, bool upd)
{
    const int cap = D.cap;
    for (unsigned long long fresh = mown & ~prevm; fresh; fresh &= fresh - 1ull)
        D.flag[(__ffsll((long long)fresh) - 1) * cap + k] |= 5;   // CONTACT_NORMAL_MODEL | CONTACT_TANGENTIAL_MODEL
    if (!upd) return;
    unsigned long long stopped = prevm & ~mown;
    while (stopped) {
        const int s = __ffsll((long long)stopped) - 1;
        stopped &= stopped - 1ull;
        D.hist_out[s * cap + k] = ldrec(&D.hist[s * cap + k]);
    }
    D.prevmask[k] = mown;
}

// The per-atom end of the step once the pair sums are in acc, for an atom
// without wall or serial work (tail_atom is false): of the post_force
// fixes only gravity acts, then FixNVESphere::final_integrate and -- when
// the run continues -- the next step's initial_integrate with the
// displacement test.
template <bool SPLIT>
__device__ __forceinline__ void atom_fix_tail(const Dev &D, int k, const dbl4 &pk, dbl4 vi4, dbl4 wi4,
                                              const dbl4 &hold, int integrate, int fuse_next, int store_f,
                                              ContactOut &acc)
{
    for (int q = 0; q < D.nfix; q++) {
        const FixDev &F = D.fix[q];
        if (F.kind == FIX_GRAVITY) {
            const double massone = vi4.w * 1.;
            acc.F[0] += massone * F.acc[0];
            acc.F[1] += massone * F.acc[1];
            acc.F[2] += massone * F.acc[2];
        }
    }
    atom_store_integrate<SPLIT>(D, k, pk, vi4, wi4, hold, integrate, fuse_next, store_f, acc);
}

// The pair step: PairGran::compute for one owned atom k with its j-side
// (reverse) entries and its own half-list entries, the post_force fixes,
// FixNVESphere::final_integrate and -- when the run continues -- the next
// step's initial_integrate with the displacement check.
//
// Shear history is double-buffered.  Invariant: when a step starts, every
// slot's current shear is in `hist` (the read buffer); the step writes the
// write buffer `hist_out`, which becomes the read buffer of the next step.
// A touching slot is read from hist and its update written to hist_out; a
// slot that stopped touching this step is copied once (after that both
// buffers agree); a rebuild writes both buffers.  Reverse entries therefore
// read the pre-update shear without racing the owner's update, exactly as
// the reference evaluates the pair once before the owner's shear changes.
//
// Per warp, the touching entries of its 32 atoms are enumerated owner-major
// (reverse entries in ascending owner order, then own entries in list
// order), evaluated one per lane in rounds of 32 with results staged in
// shared memory, and summed by each owner lane in that order.  Atoms with
// more than 64 reverse or own entries are left to the tail kernel.
template <bool ROLLING, int MINB, bool SPLIT, bool ONE, int G>
__global__ void __launch_bounds__(128, MINB) k_pair_step(Dev D, int shearupdate, int integrate, int fuse_next,
                                                         int store_f)
{
    using Real = typename std::conditional<SPLIT, float, double>::type;
    __shared__ Real sres[4][6][32];   // component-major: the owners' reads and the items' writes spread over the banks
    // the atom's records that only the tail needs (velocity, angular
    // velocity, position at the last rebuild) wait here, not in registers,
    // while the screening and the contact rounds run
    __shared__ __align__(16) dbl4 stail[3][128];
    // per warp: the touching entries listed by the screening (rev, own; the
    // launch gives 4 x 2 x D.item_cap of them in dynamic shared memory) and
    // each round's owner-lane masks, tagged with the round
    extern __shared__ __align__(16) unsigned char pair_dyn[];
    __shared__ unsigned long long sgrp[4][32];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const int k = (blockIdx.x * blockDim.x + threadIdx.x) / G;   // G lanes per atom, the first owns it
    const int wbase = (blockIdx.x * blockDim.x + wid * 32) / G;
    const bool valid = k < D.nlocal, owns = valid && (G == 1 || lane % G == 0);
    const int cap = D.cap;
    const bool upd = shearupdate != 0;
    dbl4 pk;
    unsigned long long prevm = 0ull;
    int nr = 0, nn = 0;
    unsigned long long mrev = 0ull, mown = 0ull;
    bool serial = false, tail = false;
    // what changes only at a build is read while the previous step's tail
    // kernel still runs (this grid is its programmatic dependent; the host
    // synchronises behind a build before it launches the next pair step)
    if (valid) {
        nr = D.rnum[k];
        nn = D.nnum[k];
        tail = D.tflag[k] != 0;
        serial = nr > 64 || nn > 64;
    }
    grid_dep_wait();
    grid_dep_launch();   // the tail kernel may be scheduled once every block of this grid runs
    if (step_cancelled(D)) return;
    if (valid) {
        // the atom's own records, including those only the tail needs, are
        // requested first so their latency overlaps the screening
        if (owns) {
            stage4(&stail[0][threadIdx.x], &D.vel[k]);
            stage4(&stail[1][threadIdx.x], &D.omg[k]);
            if (fuse_next) stage4(&stail[2][threadIdx.x], &D.xhold[k]);
        }
        pk = D.pos[k];
        if (!serial && upd) prevm = D.prevmask[k];
    }
    // screening of every non-serial atom of the warp, listing its touching
    // entries (all lanes take part in the list ballots)
    int nlrev = 0, nlown = 0;
    int2 *lrev = reinterpret_cast<int2 *>(pair_dyn) + (size_t)wid * 2 * D.item_cap, *lown = lrev + D.item_cap;
    const bool listed = screen_list<G, SPLIT ? 2 : 4>(D, k, (valid && !serial) ? nr : 0, (valid && !serial) ? nn : 0,
                                                      pk, mrev, mown, lrev, lown, nlrev, nlown);
    if (!listed && lane == 0 && D.item_cap > 0) atomicAdd(&D.need[4], 1);   // lists too short: counted for the host
    // FP64 path: plain in-order sums (bit-exact).  Split path: FP32 sums of
    // the FP32 pair contributions with Kahan compensation kc.
    Real as[6], kc[6];
#pragma unroll
    for (int c = 0; c < 6; c++) as[c] = kc[c] = Real(0);
    if (listed) {
        // rounds over the listed items, the rev list followed by the own list
        // (a round may hold both): lane t evaluates item base + t; the lanes
        // holding one owner's items find each other with a match, the first
        // of them publishes the group to the owner, and the owner adds its
        // items in list order
        sgrp[wid][lane] = ~0ull;
        __syncwarp();
        const int tot = nlrev + nlown;
        int round = 0;
        for (int base = 0; base < tot; base += 32, round++) {
            const int w = base + lane;
            int L = -1 - lane;   // lanes without an item match nobody
            // the next round's records on their way to L1 while this round's
            // arithmetic runs (bed of 2M spheres 847 -> 815 us/step, 1M hopper
            // unchanged; the same from the screening loop, or to L2 only, evicts
            // what the current round needs)
            if (w + 32 < tot) {
                const bool own = w + 32 >= nlrev;
                const int2 item = own ? lown[w + 32 - nlrev] : lrev[w + 32];
                const int hrow = own ? wbase + (item.y & 31) / G : item.x;
                if constexpr (SPLIT) {
                    prefetch_l1(&D.kin[item.x]);
                } else {
                    prefetch_l1(&D.vel[item.x]);
                    prefetch_l1(&D.omg[item.x]);
                }
                prefetch_l1(&D.hist[(item.y >> 8) * cap + hrow]);
            }
            if (w < tot) {
                const bool own = w >= nlrev;
                const int2 item = own ? lown[w - nlrev] : lrev[w];
                L = item.y & 31;
                Real res[6];
                eval_item<ROLLING, SPLIT, ONE>(D, wbase + L / G, item.x, item.y >> 8, own, upd, res);
#pragma unroll
                for (int c = 0; c < 6; c++) sres[wid][c][lane] = res[c];
            }
            const unsigned grp = __match_any_sync(0xffffffffu, L);
            if (w < tot && (grp & ((1u << lane) - 1u)) == 0u)
                sgrp[wid][L] = ((unsigned long long)(unsigned)round << 32) | grp;
            __syncwarp();
            const unsigned long long g = sgrp[wid][lane];
            unsigned mine = (unsigned)(g >> 32) == (unsigned)round ? (unsigned)g : 0u;
            while (mine) {
                const int q = __ffs(mine) - 1;
                mine &= mine - 1u;
                sum_item<SPLIT>(as, kc, &sres[wid][0][q]);
            }
            __syncwarp();
        }
    } else {   // a list outgrew its capacity: enumerate the bitmasks
        const int crev = __popcll(mrev);
        const WarpItems it = warp_items_cnt(owns ? crev + __popcll(mown) : 0);
        for (int base = 0; base < it.total; base += 32) {
            const int w = base + lane;
            const int L = item_owner(w, it.excl);
            const int exL = __shfl_sync(0xffffffffu, it.excl, L);
            const unsigned long long mrL = shfl64(mrev, L);
            const unsigned long long moL = shfl64(mown, L);
            if (w < it.total) {
                const int kk = wbase + L / G;
                const int q = w - exL;
                const int qr = __popcll(mrL);
                int other, s;
                bool own;
                if (q < qr) {
                    const int r = nth_set_bit(mrL, q);
                    other = __ldg(&D.rev[r * cap + kk]);
                    s = D.revs[r * cap + kk];
                    own = false;
                } else {
                    s = nth_set_bit(moL, q - qr);
                    other = __ldg(&D.nbr[s * cap + kk]);
                    own = true;
                }
                Real res[6];
                eval_item<ROLLING, SPLIT, ONE>(D, kk, other, s, own, upd, res);
#pragma unroll
                for (int c = 0; c < 6; c++) sres[wid][c][lane] = res[c];
            }
            __syncwarp();
            const int lo = max(it.excl, base), hi = min(it.excl + it.cnt, base + 32);
            for (int q = lo; q < hi; q++) sum_item<SPLIT>(as, kc, &sres[wid][0][q - base]);
            __syncwarp();
        }
    }
    ContactOut acc;
    pair_total<SPLIT>(as, kc, acc);
    if (!owns) return;
    pk = ldrec(&D.pos[k]);   // again: the rounds need its registers (packed 1M hopper 260 -> 240 us/step)
    cp_async_wait();
    if (!serial) atom_hist_tail(D, k, prevm, mown, upd);
    if (tail) {   // finished by k_pair_tail from these pair sums
        D.tailf[k] = dbl4{acc.F[0], acc.F[1], acc.F[2], 0.0};
        D.tailt[k] = dbl4{acc.T[0], acc.T[1], acc.T[2], 0.0};
        return;
    }
    const dbl4 vi4 = stail[0][threadIdx.x], wi4 = stail[1][threadIdx.x];
    dbl4 hold;
    if (fuse_next) hold = stail[2][threadIdx.x];
    atom_fix_tail<SPLIT>(D, k, pk, vi4, wi4, hold, integrate, fuse_next, store_f, acc);
}

// Second kernel of the step: the atoms listed at the last neighbour build
// as having wall candidates or more than 64 entries on a side, kTailAtoms
// per warp.  Launched as a programmatic dependent of k_pair_step, it starts
// while the pair step's last blocks run: the wall contacts of an atom with
// one wall fix at work depend only on the step's input state and that
// wall's contact history, so they are evaluated first (mesh candidates
// spread over the lanes, slot partners staged in shared memory) and their
// forces kept as records.  After the wait, each atom is finished from the
// pair sums k_pair_step left in tailf/tailt (the pairs of an atom with more
// than 64 entries on a side are evaluated here, before the wait): the
// post_force fixes in definition order with the records added at their
// fix, walls not yet done evaluated now, then final_integrate and the
// fused next initial_integrate.  Every atom's end of step touches only that
// atom's records, so the result is bit for bit that of one kernel.
// LONG: some atom of the context has more than 64 entries on a side.  The call
// of long_atom costs the kernel 1,600 bytes of spills, taken or not (a launch on
// the timed 1M hopper 30.4 us against 27.6 without it, a step of the 6,000-sphere
// hopper 20.0 against 18.9, of the 40,000-sphere drum 24.6 against 24.3), so
// contexts without such an atom, as most are, run the kernel that does not hold it.
template <bool ROLLING, bool SPLIT, bool LONG>
__global__ void __launch_bounds__(128, 4) k_pair_tail(const __grid_constant__ Dev D, int shearupdate, int integrate,
                                                      int fuse_next, int store_f)
{
    __shared__ int s_sp[4][kTailAtoms * 64];            // slot partners of the warp's atoms (mesh walls)
    __shared__ WallRec s_rec[4][kTailAtoms][kWallRec];  // wall-contact records of the warp's atoms
    // every thread waits for the pair step before it exits, so this grid's
    // completion implies the pair step's for the launches after it
    if (step_cancelled(D)) {
        grid_dep_wait();
        return;
    }
    const int n = *D.tailcnt;
    const bool upd = shearupdate != 0;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const int nwarp = gridDim.x * (blockDim.x >> 5);
    WallRec *rec = s_rec[wid][lane < kTailAtoms ? lane : 0];
    for (int base = (blockIdx.x * (blockDim.x >> 5) + wid) * kTailAtoms; base < n; base += nwarp * kTailAtoms) {
        const bool own = lane < kTailAtoms && base + lane < n;
        int i = 0, ti = 0, nr = 0, nn = 0, qw = -1, nwork = 0;
        dbl4 pi, vi4, wi4, hold;
        pi = vi4 = wi4 = hold = dbl4{0.0, 0.0, 0.0, 0.0};
        if (own) {
            i = D.tail[base + lane];
            pi = ldrec_l2(&D.pos[i]);
            vi4 = ldrec_l2(&D.vel[i]);
            wi4 = ldrec_l2(&D.omg[i]);
            if (fuse_next) hold = D.xhold[i];
            ti = D.type[i];
            nr = D.rnum[i];
            nn = D.nnum[i];
            for (int q = 0; q < D.nfix; q++) {
                const FixDev &F = D.fix[q];
                if ((F.kind == FIX_WALL_PLANE && F.inlist[i]) || (F.kind == FIX_WALL_MESH && F.mesh.tcnt[i] != 0)) {
                    qw = q;
                    nwork++;
                }
            }
        }
        const bool serial = LONG && (nr > 64 || nn > 64);
        // long lists, also before the wait: their sums need nothing of the pair step
        ContactOut lacc;
        for (int c = 0; c < 3; c++) lacc.F[c] = lacc.T[c] = 0.0;
        if constexpr (LONG)
            for (unsigned m = __ballot_sync(0xffffffffu, own && serial); m; m &= m - 1u) {
                const int src = __ffs(m) - 1;
                ContactOut a;
                long_atom<ROLLING>(D, __shfl_sync(0xffffffffu, i, src), __shfl_sync(0xffffffffu, nr, src),
                                   __shfl_sync(0xffffffffu, nn, src), upd, s_sp[wid], a);
                if (lane == src) {
                    lacc = a;
                    if (upd) D.prevmask[i] = ~0ull;   // every own slot written this step
                }
            }
        const double vi[3] = {vi4.x, vi4.y, vi4.z}, wi[3] = {wi4.x, wi4.y, wi4.z};
        // walls before the wait: atoms with one wall fix at work
        bool early = own && !serial && nwork == 1;
        int nrec = 0;
        ContactOut unused;
        for (int q = 0; q < D.nfix; q++) {
            const FixDev &F = D.fix[q];
            if (F.kind == FIX_WALL_PLANE) {
                if (early && qw == q) {
                    ContactOut o = wall_record_zero();
                    if (plane_wall_atom(D, F, i, pi, vi, wi, vi4.w, ti, upd, o)) wall_record_put(rec, nrec, o);
                }
            } else if (F.kind == FIX_WALL_MESH && __any_sync(0xffffffffu, early && qw == q)) {
                mesh_wall_items<true>(D, F.mesh, early && qw == q, i, pi, vi, wi, vi4.w, ti, upd, s_sp[wid], unused,
                                      rec, &nrec, &early);
            }
        }
        grid_dep_wait();
        grid_dep_launch();   // the next step's pair step may be scheduled (it waits for this grid)
        ContactOut acc;
        for (int c = 0; c < 3; c++) acc.F[c] = acc.T[c] = 0.0;
        if (own) {
            if (serial) {
                acc = lacc;
            } else {
                const dbl4 F4 = D.tailf[i], T4 = D.tailt[i];
                acc.F[0] = F4.x;
                acc.F[1] = F4.y;
                acc.F[2] = F4.z;
                acc.T[0] = T4.x;
                acc.T[1] = T4.y;
                acc.T[2] = T4.z;
            }
        }
        const bool late = own && !early;   // walls evaluated after the wait
        for (int q = 0; q < D.nfix; q++) {
            const FixDev &F = D.fix[q];
            if (F.kind == FIX_GRAVITY) {
                const double massone = vi4.w * 1.;
                acc.F[0] += massone * F.acc[0];
                acc.F[1] += massone * F.acc[1];
                acc.F[2] += massone * F.acc[2];
            } else if (F.kind == FIX_WALL_PLANE || F.kind == FIX_WALL_MESH) {
                if (early && qw == q) {   // this fix's records, in the order they were made
                    for (int r = 0; r < nrec; r++) {
                        acc.F[0] += rec[r][0];
                        acc.F[1] += rec[r][1];
                        acc.F[2] += rec[r][2];
                        acc.T[0] += rec[r][3];
                        acc.T[1] += rec[r][4];
                        acc.T[2] += rec[r][5];
                    }
                }
                // walls left for now; the mesh routine is warp-collective, so
                // every lane calls it (owners without work pass own = false)
                if (F.kind == FIX_WALL_PLANE) {
                    if (late && F.inlist[i]) plane_wall_atom(D, F, i, pi, vi, wi, vi4.w, ti, upd, acc);
                } else if (__any_sync(0xffffffffu, late)) {
                    mesh_wall_items<false>(D, F.mesh, late, i, pi, vi, wi, vi4.w, ti, upd, s_sp[wid], acc);
                }
            }
        }
        if (own) atom_store_integrate<SPLIT>(D, i, pi, vi4, wi4, hold, integrate, fuse_next, store_f, acc);
    }
    grid_dep_wait();
}

// Host side: a kernel launched as a programmatic dependent of the one before it
// on the same stream.
template <typename Kernel>
inline cudaError_t launch_dependent(Kernel kernel, int nblocks, size_t smem, cudaStream_t st, const Dev &D,
                                    int shearupdate, int integrate, int fuse_next, int store_f)
{
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(nblocks);
    cfg.blockDim = dim3(128);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kernel, D, shearupdate, integrate, fuse_next, store_f);
}

// The pair step with one or (FP64) two lanes per atom.  Registers: FP64 takes 4 blocks
// per SM (128 registers, at most 4 bytes of spills): 5 blocks (96) spill 20
// doubles through the L1 that the gathers need, 3 leave too few warps (hopper of
// 1M 253, 267 and 307 us/step, bed of 2M 847, 907 and 847).  Split precision takes
// 6 blocks (80, with 40 to 68 bytes spilled): 206 us/step against 209 with 5 and
// 240 with 4.
template <bool ROLLING, bool SPLIT, bool ONE>
inline cudaError_t launch_pair_one(const Dev &D, int lanes, cudaStream_t st, int shearupdate, int integrate,
                                   int fuse_next, int store_f, size_t smem)
{
    auto kernel = k_pair_step<ROLLING, SPLIT ? 6 : 4, SPLIT, ONE, 1>;
    if constexpr (!SPLIT) {
        if (lanes == 2) kernel = k_pair_step<ROLLING, 4, false, ONE, 2>;
    }
    const int nblocks = (int)(((long)D.nlocal * lanes + 127) / 128);
    return launch_dependent(kernel, nblocks, smem, st, D, shearupdate, integrate, fuse_next, store_f);
}

template <bool SPLIT>
inline cudaError_t launch_pair_step(const Dev &D, int lanes, cudaStream_t st, int shearupdate, int integrate,
                                    int fuse_next, int store_f, size_t smem)
{
    if (D.rolling && D.ntypes == 1)
        return launch_pair_one<true, SPLIT, true>(D, lanes, st, shearupdate, integrate, fuse_next, store_f, smem);
    if (D.rolling)
        return launch_pair_one<true, SPLIT, false>(D, lanes, st, shearupdate, integrate, fuse_next, store_f, smem);
    if (D.ntypes == 1)
        return launch_pair_one<false, SPLIT, true>(D, lanes, st, shearupdate, integrate, fuse_next, store_f, smem);
    return launch_pair_one<false, SPLIT, false>(D, lanes, st, shearupdate, integrate, fuse_next, store_f, smem);
}

// Host side: the tail kernel of the pair step launched just before it.
template <bool SPLIT>
inline cudaError_t launch_pair_tail(const Dev &D, bool long_lists, int nblocks, cudaStream_t st, int shearupdate,
                                    int integrate, int fuse_next, int store_f)
{
    auto kernel = k_pair_tail<false, SPLIT, false>;
    if (D.rolling && long_lists) kernel = k_pair_tail<true, SPLIT, true>;
    else if (D.rolling) kernel = k_pair_tail<true, SPLIT, false>;
    else if (long_lists) kernel = k_pair_tail<false, SPLIT, true>;
    return launch_dependent(kernel, nblocks, 0, st, D, shearupdate, integrate, fuse_next, store_f);
}

}  // namespace gb2
