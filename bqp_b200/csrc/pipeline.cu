// Stage-synchronous propagation engine.
//
// The persistent kernel (propagate.cu) runs the whole force model and the
// controller inside one thread per trajectory; at 70x70 + JB2008 that kernel
// is large, register-bound (255 registers, 8 warps per SM) and stalls on
// instruction fetch.  Here every RK stage of every active trajectory is one
// pass over three specialised kernels, and one controller kernel closes the
// attempt:
//
//   pl_times<M>     for several stages at once, what depends on a stage's
//                   instant alone: Kepler baseline, Earth rotation, Sun, Moon
//                                                           (FP64 latency bound)
//   pl_prep<M>(s)   finish stage s-1, form y_s = y + h sum a_sj k_j, third body
//                   and Battin's term                       (load latency bound)
//   pl_gravity      normalised column recursion, table in shared memory
//                                                           (FP64-FMA bound)
//   pl_drag         JB2008 density and co-rotating drag     (transcendental bound)
//   pl_control<M>   finish the last stage, error norm, accept / reject, samples,
//                   rectification, next attempt; compacts the active list
//
// Stage data are indexed by the trajectory's slot in the active list, so the
// force kernels stream contiguous arrays; the active list shrinks as
// trajectories finish.  The attempt sequence is captured once as a CUDA graph
// and replayed; the host reads the active count between replays.
#include <cuda_runtime.h>

#include <algorithm>
#include <chrono>
#include <cstdint>
#include <vector>

#include "kernels.cuh"
#include "launch.h"
#include "traj.cuh"

namespace bqp {

namespace {

constexpr int kBlock = 256;

// Drag lanes per state above and below ~510 km (the lanes share the sweep
// series and the intervals walked exactly), and the drag kernel's minimum
// resident CTAs per SM, which sets its register budget.  The stage's drag runs
// beside its gravity, which leaves it half of an SM's registers (128 threads
// of 248): 65,536 rows at 70x70, exact model, us a pass: 327,168 with 80
// registers (6 CTAs of 128), 332,036 with 64, 333,552 with 96, 331,616 with
// 128; one after the other 398,180.  Where all rows fit in a wave anyway, 128
// registers and no spills: 7,000 rows 188,420 us against 207,638.
#ifndef BQP_DRAG_LANES_HIGH
#define BQP_DRAG_LANES_HIGH 1
#endif
#ifndef BQP_DRAG_LANES_LOW
#define BQP_DRAG_LANES_LOW 4
#endif
#ifndef BQP_DRAG_MIN_BLOCKS
#define BQP_DRAG_MIN_BLOCKS 6
#endif
#ifndef BQP_DRAG_MIN_BLOCKS_FEW
#define BQP_DRAG_MIN_BLOCKS_FEW 4
#endif
#ifndef BQP_DRAG_BLOCK
#define BQP_DRAG_BLOCK 128
#endif
constexpr int kDragBlock = BQP_DRAG_BLOCK;
// stage derivative buffers per row: the most stages of any tableau (Vern9's
// 16) plus the dense-output stage of the sampled non-FSAL path
constexpr int kStageBufs = Tab<kVern9>::S + 1;

__device__ __forceinline__ double* K(const PipeBufs& P, int st, int i) { return P.k + ((size_t)st * 6 + i) * P.cap; }

// Append `traj` to the next active list (warp-aggregated atomic).
__device__ __forceinline__ void append_active(int32_t* list, int32_t* count, int32_t traj, bool keep) {
    const unsigned mask = __ballot_sync(0xffffffffu, keep);
    if (!keep) return;
    const int lane = threadIdx.x & 31;
    const int leader = __ffs(mask) - 1;
    int base = 0;
    if (lane == leader) base = atomicAdd(count, __popc(mask));
    base = __shfl_sync(mask, base, leader);
    const int rank = __popc(mask & ((1u << lane) - 1u));
    list[base + rank] = traj;
}

// What stage `st` needs of its instant, in the ring.
struct StageTimes {
    double* p;
    int64_t cap;
    __device__ __forceinline__ StageTimes(const PipeBufs& P, int st)
        : p(P.tq + (size_t)(st % P.ring) * P.fields * P.cap), cap(P.cap) {}
    __device__ __forceinline__ double& at(int field, int slot) const { return p[(size_t)field * cap + slot]; }
    __device__ __forceinline__ double& baseline(int i, int slot) const { return at(i, slot); }
    __device__ __forceinline__ double& sun(int i, int slot) const { return at(6 + i, slot); }
    __device__ __forceinline__ double& moon(int i, int slot) const { return at(9 + i, slot); }
    __device__ __forceinline__ double& jd(int slot) const { return at(12, slot); }
    // GMST: sin, cos; IAU: R (row-major) and the ITRS angular velocity (GCRS)
    __device__ __forceinline__ double& frame(int i, int slot) const { return at(13 + i, slot); }
    // with drag, the last six: the Sun's Earth-fixed x and y, its declination,
    // and jb::EpochR (tsubc NaN: no or invalid drivers)
    __device__ __forceinline__ double& drag(const PipeBufs& P, int i, int slot) const {
        return at(P.fields - 6 + i, slot);
    }
};
constexpr int kTimesFields = 13, kTimesGmst = 2, kTimesIau = 12, kTimesDrag = 6;

// Sum of the stage-`st` force terms into K(st, 3..5).
__device__ __forceinline__ void finish_stage(const PipeBufs& P, int st, int slot) {
    const StageTimes T(P, st);
    const double gx = P.agrav[slot], gy = P.agrav[P.cap + slot], gz = P.agrav[2 * P.cap + slot];
    if (P.iau) {
        double r[9], g[3];
        const double gi[3] = {gx, gy, gz};
        for (int e = 0; e < 9; ++e) r[e] = T.frame(e, slot);
        ft::to_gcrs(r, gi, g);
        for (int i = 0; i < 3; ++i)
            K(P, st, 3 + i)[slot] = g[i] + P.adrag[(size_t)i * P.cap + slot] + P.part[(size_t)i * P.cap + slot];
        return;
    }
    const double s = T.frame(0, slot), c = T.frame(1, slot);
    K(P, st, 3)[slot] = fma(c, gx, -s * gy) + P.adrag[slot] + P.part[slot];
    K(P, st, 4)[slot] = fma(s, gx, c * gy) + P.adrag[P.cap + slot] + P.part[P.cap + slot];
    K(P, st, 5)[slot] = gz + P.adrag[2 * P.cap + slot] + P.part[2 * P.cap + slot];
}

// An ECI vector of slot `slot` in the Earth-fixed frame of stage T.
__device__ __forceinline__ void slot_to_itrs(const PipeBufs& P, const StageTimes& T, int slot, const double* v,
                                             double* o) {
    if (P.iau) {
        double r[9];
        for (int e = 0; e < 9; ++e) r[e] = T.frame(e, slot);
        ft::to_itrs(r, v, o);
    } else {
        const double s = T.frame(0, slot), c = T.frame(1, slot);
        o[0] = fma(c, v[0], s * v[1]);
        o[1] = fma(-s, v[0], c * v[1]);
        o[2] = v[2];
    }
}

}  // namespace

// --------------------------------------------------------------------- init
template <int M>
__global__ void __launch_bounds__(kBlock) pl_init(PropArgs A, PipeBufs P) {
    const int64_t traj = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    bool keep = false;
    if (traj < A.n) {
        TrajState s;
        traj_begin(A, s, traj);
        if (s.phase == kNeedSegment) seg_begin<M>(A, s, traj);
        if (s.phase == kStepping) {
            const int32_t f = attempt_begin<M>(A, s, false);
            if (f >= 0) traj_fail(A, s, traj, f);
            else keep = true;
        }
        P.st[traj] = s;
    }
    append_active(P.idx[0], &P.count[0], (int32_t)traj, keep);
}

// -------------------------------------------------------------------- times
// Stages st0 .. st0 + gridDim.y - 1 of the current attempt, one stage of one
// row a thread.  st == S is the dense-output stage of the sampled non-FSAL
// path: f(t_next, y_next) evaluated before the controller decides (the
// reference evaluates it after an accept).
//
// Everything here is known when the attempt begins, so the stages' long FP64
// chains (the Kepler solve, the Sun and Moon series, the frame) run side by
// side once an attempt instead of one after the other before each stage's
// force.
template <int M>
__global__ void __launch_bounds__(kBlock) pl_times(PropArgs A, PipeBufs P, int cur, int st0) {
    using T = Tab<M>;
    const int slot = blockIdx.x * blockDim.x + threadIdx.x, st = st0 + blockIdx.y;
    if (blockIdx.x == 0 && threadIdx.x < 2) P.dcount[2 * (st % P.ring) + threadIdx.x] = 0;
    if (slot >= P.count[cur]) return;
    const TrajState& s = P.st[P.idx[cur][slot]];
    if (st == 0 && (s.flags & kHaveK1)) return;
    const StageTimes Q(P, st);
    const double ts = st < T::S ? s.t + T::c(st) * s.hs : next_time(s);
    double rs[6];
    baseline_state(baseline_new(s.cur), ts - s.ct0, rs);
    for (int i = 0; i < 6; ++i) Q.baseline(i, slot) = rs[i];
    const double jd = utc_jd_at(s.jd0, ts);
    Q.jd(slot) = jd;
    const ForceParams& fp = A.force;
    if (P.iau) {
        // the IAU 2006/2000A rotation of the stage's instant (rhs.rs:3113-3174);
        // NaN where it has none
        ft::FrameRot F;
        if ((fp.gravity_on || fp.drag) && !frame_rot(fp.frame, s.tai0 + ts, F)) {
            for (int e = 0; e < 9; ++e) F.r[e] = NAN;
            F.w[0] = F.w[1] = F.w[2] = NAN;
        } else if (!(fp.gravity_on || fp.drag)) {
            for (int e = 0; e < 9; ++e) F.r[e] = (e % 4 == 0) ? 1.0 : 0.0;
            F.w[0] = F.w[1] = F.w[2] = 0.0;
        }
        for (int e = 0; e < 9; ++e) Q.frame(e, slot) = F.r[e];
        for (int e = 0; e < 3; ++e) Q.frame(9 + e, slot) = F.w[e];
    } else {
        double sn = 0.0, cs = 1.0;
        if (fp.gravity_on || fp.drag) sincos(gmst_rad(jd), &sn, &cs);
        Q.frame(0, slot) = sn;
        Q.frame(1, slot) = cs;
    }
    if (fp.sun || (fp.drag && s.cd != 0.0 && s.am != 0.0) || s.side >= 0) {
        double sun[3];
        sun_at(fp.eph_sun, jd, sun);
        for (int i = 0; i < 3; ++i) Q.sun(i, slot) = sun[i];
        if (fp.drag) {
            // JB2008 adapter (rhs.rs:3551-3776), as Encke::density_at: the
            // Sun's side of it and the drivers'
            double si[3];
            slot_to_itrs(P, Q, slot, sun, si);
            const double sun_r = sqrt(fma(si[0], si[0], fma(si[1], si[1], si[2] * si[2])));
            Q.drag(P, 0, slot) = si[0];
            Q.drag(P, 1, slot) = si[1];
            Q.drag(P, 2, slot) = asin(fmin(1.0, fmax(-1.0, si[2] / sun_r)));
            jb::Drivers dr = fp.drivers;
            const double mjd = jd - 2400000.5;
            double tsubc = NAN, sinphi = 0.0, gtz = 0.0;
            if ((fp.dtab.n_solar == 0 || jb::lookup_drivers(fp.dtab, jd, &dr)) && jb::drivers_valid(mjd, dr)) {
                if (fp.drag_fp32) {
                    const jb::EpochR<float> E = jb::epoch_terms<float>(mjd, dr, true);
                    tsubc = E.tsubc;
                    sinphi = E.sinphi;
                    gtz = E.gtz;
                } else {
                    const jb::EpochR<double> E = jb::epoch_terms<double>(mjd, dr, fp.atm_model != 4);
                    tsubc = E.tsubc;
                    sinphi = E.sinphi;
                    gtz = E.gtz;
                }
            }
            Q.drag(P, 3, slot) = tsubc;
            Q.drag(P, 4, slot) = sinphi;
            Q.drag(P, 5, slot) = gtz;
        }
    }
    if (fp.moon) {
        double moon[3];
        moon_at(fp.eph_moon, jd, moon);
        for (int i = 0; i < 3; ++i) Q.moon(i, slot) = moon[i];
    }
}

// --------------------------------------------------------------------- prep
template <int M>
__global__ void __launch_bounds__(kBlock) pl_prep(PropArgs A, PipeBufs P, int cur, int st) {
    using T = Tab<M>;
    const int slot = blockIdx.x * blockDim.x + threadIdx.x;
    if (st == 0 && blockIdx.x == 0 && threadIdx.x == 0) P.count[cur ^ 1] = 0;
    if (slot >= P.count[cur]) return;
    const int32_t traj = P.idx[cur][slot];
    const TrajState& s = P.st[traj];
    if (st == 0) {
        P.bad[slot] = 0;
        if (s.flags & kHaveK1) {
            for (int i = 0; i < 6; ++i) K(P, 0, i)[slot] = s.k1c[i];
            P.skip[slot] = 1;
            return;
        }
    } else if (!(st == 1 && P.skip[slot])) {
        finish_stage(P, st - 1, slot);
    }
    P.skip[slot] = 0;
    // stage state
    double yt[6];
    for (int i = 0; i < 6; ++i) yt[i] = s.y[i];
    if (st < T::S) {
#pragma unroll 1
        for (int j = 0; j < st; ++j) {
            const double a = s.hs * T::a(st, j);
            if (a != 0.0)
                for (int i = 0; i < 6; ++i) yt[i] = fma(K(P, j, i)[slot], a, yt[i]);
        }
    } else {
        // y_next exactly as rk_combine forms it
#pragma unroll 1
        for (int j = 0; j < T::S; ++j) {
            const double b = s.hs * T::b(j);
            if (b != 0.0)
                for (int i = 0; i < 6; ++i) yt[i] = fma(K(P, j, i)[slot], b, yt[i]);
        }
    }
    const StageTimes Q(P, st);
    double rs[6], sp[6];
    for (int i = 0; i < 6; ++i) {
        rs[i] = Q.baseline(i, slot);
        sp[i] = rs[i] + yt[i];
        P.sp[(size_t)i * P.cap + slot] = sp[i];
    }
    for (int i = 0; i < 3; ++i) K(P, st, i)[slot] = yt[3 + i];
    const ForceParams& fp = A.force;
    if (P.iau && (fp.gravity_on || fp.drag) && isnan(Q.frame(0, slot))) P.bad[slot] = 3;
    double acc[3] = {0.0, 0.0, 0.0};
    double sun[3];
    const bool need_sun = fp.sun || (fp.drag && s.cd != 0.0 && s.am != 0.0) || s.side >= 0;
    if (need_sun)
        for (int i = 0; i < 3; ++i) sun[i] = Q.sun(i, slot);
    if (s.side >= 0) srp_accel(sp, sun, fp.p_sun, fp.cr, s.am, s.side, acc);  // on the leg's fixed side
    if (fp.sun) third_body(sp, sun, fp.mu_sun, acc);
    if (fp.moon) {
        const double moon[3] = {Q.moon(0, slot), Q.moon(1, slot), Q.moon(2, slot)};
        third_body(sp, moon, fp.mu_moon, acc);
    }
    const double r2 = fma(sp[0], sp[0], fma(sp[1], sp[1], sp[2] * sp[2]));
    battin(rs, yt, r2, sqrt(r2), acc);
    for (int i = 0; i < 3; ++i) P.part[(size_t)i * P.cap + slot] = acc[i];
    if (fp.drag) {
        P.amcd[slot] = s.am;
        P.amcd[P.cap + slot] = s.cd;
        // drag work list: states above ~510 km take the sweep fits (cheap),
        // the rest walk the quadrature; homogeneous warps in each list
        const int cls = sqrt(r2) - fp.earth_radius >= 510.0 ? 0 : 1;
        const unsigned m = __activemask();
#pragma unroll
        for (int c = 0; c < 2; ++c) {
            const unsigned mm = __ballot_sync(m, cls == c);
            if (cls == c) {
                const int lane = threadIdx.x & 31;
                const int leader = __ffs(mm) - 1;
                int base = 0;
                if (lane == leader) base = atomicAdd(&P.dcount[2 * (st % P.ring) + c], __popc(mm));
                base = __shfl_sync(mm, base, leader);
                P.dlist[c][base + __popc(mm & ((1u << lane) - 1u))] = slot;
            }
        }
    } else {
        for (int i = 0; i < 3; ++i) P.adrag[(size_t)i * P.cap + slot] = 0.0;
    }
    if (!fp.gravity_on)
        for (int i = 0; i < 3; ++i) P.agrav[(size_t)i * P.cap + slot] = 0.0;
}

// ------------------------------------------------------------------ gravity
// Persistent over slots: every CTA (or cluster) takes an equal, contiguous
// share of the active slots.
// `out` receives the field; with `list` set the rows are the slots
// list[0 .. *list_count) instead of the active slots 0 .. count.
template <int NT, int kForm>
__global__ void __launch_bounds__(256, 1) pl_gravity(const __grid_constant__ GravTable T, int aux, PipeBufs P, int cur,
                                                     int st, double* out, const int32_t* list,
                                                     const int32_t* list_count) {
    int64_t per, c0, c1;
    gravity_rows<kForm>(list ? *list_count : P.count[cur], aux, &per, &c0, &c1);
    const int b0 = (int)c0, b1 = (int)c1;
    const StageTimes Q(P, st);
    if (b0 >= b1) return;  // uniform across the CTA and its cluster
    auto load = [&](int row, double& x, double& y, double& z) -> bool {
        const int sl = list ? list[row] : row;
        if (P.skip[sl]) return false;
        const double e[3] = {P.sp[sl], P.sp[P.cap + sl], P.sp[2 * P.cap + sl]};
        double q[3];
        slot_to_itrs(P, Q, sl, e, q);
        const double r2 = fma(q[0], q[0], fma(q[1], q[1], q[2] * q[2]));
        if (!(isfinite(r2) && r2 > 0.0)) {
            if (!P.bad[sl]) P.bad[sl] = 1;
            out[sl] = out[P.cap + sl] = out[2 * P.cap + sl] = NAN;
            return false;
        }
        x = q[0];
        y = q[1];
        z = q[2];
        return true;
    };
    auto store = [&](int row, const double* a) {
        const int sl = list ? list[row] : row;
        out[sl] = a[0];
        out[P.cap + sl] = a[1];
        out[2 * P.cap + sl] = a[2];
    };
    auto lost = [&](int row) {
        const int sl = list ? list[row] : row;
        P.bad[sl] = 2;
        out[sl] = out[P.cap + sl] = out[2 * P.cap + sl] = NAN;
    };
    gravity_cta<NT, kForm>(T, aux, (int)per, b0, b1, load, store, lost);
}

using GravKernel = void (*)(const GravTable, int, PipeBufs, int, int, double*, const int32_t*, const int32_t*);

template <int F>
static GravKernel pl_gravity_form(int nt) {
    return nt == 1 ? pl_gravity<1, F> : nt == 2 ? pl_gravity<2, F> : pl_gravity<4, F>;
}

static GravKernel pl_gravity_of(const GravLaunch& G) {
    return G.form == kGravSplit     ? pl_gravity_form<kGravSplit>(G.nt)
           : G.form == kGravCluster ? pl_gravity_form<kGravCluster>(G.nt)
                                    : pl_gravity_form<kGravPlain>(G.nt);
}

// Earth-fixed positions of the stage's active slots, [slot][3] (the
// surrogate's input)
__global__ void __launch_bounds__(kBlock) pl_earth_fixed(PipeBufs P, int cur, int st) {
    const int sl = blockIdx.x * blockDim.x + threadIdx.x;
    if (sl >= P.count[cur]) return;
    const double e[3] = {P.sp[sl], P.sp[P.cap + sl], P.sp[2 * P.cap + sl]};
    slot_to_itrs(P, StageTimes(P, st), sl, e, P.ef + 3 * (size_t)sl);
}

// ------------------------------------------------------- surrogate check
// Per step, at its first stage: the network's field (agrav) against the
// exact one (agx), both without the central term.  A row off by more than
// `thr` of the whole exact field's magnitude (central term included) takes
// the exact field now and, through the slot list, at the step's later
// stages.  A row whose first stage was carried over (a retried step, or the
// FSAL stage of the step before) keeps the verdict under which that stage
// was evaluated.
__global__ void __launch_bounds__(kBlock) pl_sur_check(PipeBufs P, int cur, double thr) {
    const int sl = blockIdx.x * blockDim.x + threadIdx.x;
    if (sl >= P.count[cur]) return;
    const int32_t traj = P.idx[cur][sl];
    if (!P.skip[sl]) {
        const double* q = P.ef + 3 * (size_t)sl;  // Earth-fixed position
        const double r2 = fma(q[0], q[0], fma(q[1], q[1], q[2] * q[2]));
        const double kc = -kMu / (r2 * sqrt(r2));
        double d2 = 0.0, a2 = 0.0;
        for (int k = 0; k < 3; ++k) {
            const size_t o = (size_t)k * P.cap + sl;
            const double d = P.agrav[o] - P.agx[o];
            const double a = fma(kc, q[k], P.agx[o]);
            d2 = fma(d, d, d2);
            a2 = fma(a, a, a2);
        }
        const bool fall = !(d2 <= thr * thr * a2);  // NaN falls back too
        P.fall[traj] = fall ? 1 : 0;
        if (fall)
            for (int k = 0; k < 3; ++k) P.agrav[(size_t)k * P.cap + sl] = P.agx[(size_t)k * P.cap + sl];
    }
    if (P.fall[traj]) P.flist[atomicAdd(P.fcount, 1)] = sl;
}

// --------------------------------------------------------------------- drag
// One state per group of L lanes (jb::density_group): the JB2008 model is the
// longest serial chain of the force call, and the kernel is bound by that
// latency, not by throughput.  Both drag lists go in one launch (blocks
// [0, nb_hi) take list 0 with LH lanes per state, the rest list 1 with LL),
// so that a stage's states are resident together in as few waves as the
// register budget allows.
// kForm 0: the exact model; 1, 2: the coarse profiles in FP64 and in FP32; 3:
// the exact model in the order of PropArgs::ordered (and the profiles without
// the fixed plans' ends: plan null).
template <int L, int kForm = 0>
__device__ __forceinline__ void drag_rows(const ForceParams& fp, const PipeBufs& P, int st, int list, int block) {
    const int gt = block * blockDim.x + threadIdx.x;
    const int item = gt / L;
    const int q = gt % L;
    const unsigned gmask = ((1u << L) - 1u) << ((threadIdx.x & 31) & ~(L - 1));
    if (item >= P.dcount[2 * (st % P.ring) + list]) return;  // uniform across the group
    const int slot = P.dlist[list][item];
    double sp[6];
    for (int i = 0; i < 6; ++i) sp[i] = P.sp[(size_t)i * P.cap + slot];
    const double am = P.amcd[slot], cd = P.amcd[P.cap + slot];
    double a[3] = {0.0, 0.0, 0.0};
    if (cd != 0.0 && am != 0.0) {
        // JB2008 adapter (rhs.rs:3551-3776), as Encke::density_at
        const StageTimes Q(P, st);
        double pi[3];
        slot_to_itrs(P, Q, slot, sp, pi);
        const double sat_r = sqrt(fma(pi[0], pi[0], fma(pi[1], pi[1], pi[2] * pi[2])));
        double rho;
        if ((sat_r - fp.earth_radius) * 1000.0 > 2500.0e3) {
            rho = 1.0e-19;
        } else {
            const double si0 = Q.drag(P, 0, slot), si1 = Q.drag(P, 1, slot), dec = Q.drag(P, 2, slot);
            const jb::EpochR<double> E{Q.drag(P, 3, slot), Q.drag(P, 4, slot), Q.drag(P, 5, slot)};
            const double alt_m = geodetic_altitude_km(pi[0], pi[1], pi[2], fp.earth_radius) * 1000.0;
            const double ha = atan2(fma(pi[1], si0, -(pi[0] * si1)), fma(pi[0], si0, pi[1] * si1));
            const double lat = asin(fmin(1.0, fmax(-1.0, pi[2] / sat_r)));
            jb::Drivers dr = fp.drivers;
            if (fp.dtab.n_solar > 0) jb::lookup_drivers(fp.dtab, Q.jd(slot), &dr);
            // fixed-node fits from constant memory (fp.fit holds the same numbers);
            // no drivers at this instant -> NaN density (rhs.rs:3560-3571), the
            // same verdict on every lane of the group
            if (isnan(E.tsubc))
                rho = NAN;
            else if (kForm == 0 || kForm == 3)
                rho = jb::density_group<L, kForm == 3>(E, dec, ha, lat, alt_m, dr, q, gmask, fp.fit != nullptr,
                                                       fp.fit2);
            else if (!jb::geometry_valid(dec, ha, lat, alt_m))
                rho = NAN;
            else if (kForm == 2)
                rho = jb::density_coarse_core<float>({(float)E.tsubc, (float)E.sinphi, (float)E.gtz}, dec, ha, lat,
                                                     alt_m, dr, fp.atm_model, &fp.plan);
            else
                rho = jb::density_coarse_core<double>(E, dec, ha, lat, alt_m, dr, fp.atm_model, &fp.plan);
            if (!(rho > 0.0) || !isfinite(rho)) rho = NAN;
            else if (alt_m > 2500.0e3) rho = fmin(rho, 1.0e-19);
        }
        if (isnan(rho)) {
            a[0] = a[1] = a[2] = NAN;
        } else if (rho > 0.0) {
            double vr0, vr1, vr2;
            if (P.iau) {
                // atmosphere co-rotating with the resolved frame (rhs.rs:1134-1139)
                double w[3];
                const StageTimes Q(P, st);
                for (int e = 0; e < 3; ++e) w[e] = Q.frame(9 + e, slot);
                vr0 = (sp[3] - (w[1] * sp[2] - w[2] * sp[1])) * 1000.0;
                vr1 = (sp[4] - (w[2] * sp[0] - w[0] * sp[2])) * 1000.0;
                vr2 = (sp[5] - (w[0] * sp[1] - w[1] * sp[0])) * 1000.0;
            } else {
                const double w = fp.omega;
                vr0 = (sp[3] + w * sp[1]) * 1000.0;
                vr1 = (sp[4] - w * sp[0]) * 1000.0;
                vr2 = sp[5] * 1000.0;
            }
            const double v2 = fma(vr0, vr0, fma(vr1, vr1, vr2 * vr2));
            if (v2 != 0.0) {
                const double k = -0.5 * cd * am * rho * sqrt(v2) * 1e-3;
                a[0] = k * vr0;
                a[1] = k * vr1;
                a[2] = k * vr2;
            }
        }
    }
    if (q == 0)
        for (int i = 0; i < 3; ++i) P.adrag[(size_t)i * P.cap + slot] = a[i];
}

template <int LH, int LL, int kMinBlocks, int kForm>
__global__ void __launch_bounds__(kDragBlock, kMinBlocks) pl_drag(ForceParams fp, PipeBufs P, int st, int nb_hi) {
    if ((int)blockIdx.x < nb_hi) drag_rows<LH, kForm>(fp, P, st, 0, blockIdx.x);
    else drag_rows<LL, kForm>(fp, P, st, 1, blockIdx.x - nb_hi);
}

// The coarse profiles (atm_model 5-7): a short chain per state, one lane
// each, both altitude lists in one launch.
#ifndef BQP_COARSE_MIN_BLOCKS
#define BQP_COARSE_MIN_BLOCKS 4
#endif
template <int kForm>
__global__ void __launch_bounds__(kDragBlock, BQP_COARSE_MIN_BLOCKS) pl_drag_coarse(ForceParams fp, PipeBufs P, int st, int nb_hi) {
    if ((int)blockIdx.x < nb_hi) drag_rows<1, kForm>(fp, P, st, 0, blockIdx.x);
    else drag_rows<1, kForm>(fp, P, st, 1, blockIdx.x - nb_hi);
}

// ------------------------------------------------------------------ control
// Splits a row's own thread may take on its crossing scan before the warp
// takes it over.
#ifndef BQP_ECL_SOLO_SPLITS
#define BQP_ECL_SOLO_SPLITS 4
#endif
constexpr int64_t kEclSoloSplits = BQP_ECL_SOLO_SPLITS;

template <int M>
__global__ void __launch_bounds__(kBlock) pl_control(PropArgs A, PipeBufs P, int cur, int dense,
                                                      int timed_out) {
    using T = Tab<M>;
    // per warp: the store of the cooperative eclipse scan (SRP rows)
    __shared__ EclWarpStore ecl_ws[kBlock / 32];
    const int slot = blockIdx.x * blockDim.x + threadIdx.x;
    const int lane = threadIdx.x & 31;
    const int count = P.count[cur];
    if (slot - lane >= count) return;  // the whole warp is idle
    const bool active = slot < count;
    bool keep = false;
    int32_t traj = 0;
    TrajState s;
    bool scan = false;  // an accepted SRP step waiting for its crossing scan
    EclScanReq req;
    double tn = 0.0, en = 0.0, ynext[6], k0[6], dyn[6];
    if (active) {
        traj = P.idx[cur][slot];
        s = P.st[traj];
        const int last = dense ? T::S : T::S - 1;
        if (!(last == 1 && P.skip[slot])) finish_stage(P, last, slot);
        // stage derivatives of this attempt
        const int evaluated = T::S - ((s.flags & kHaveK1) ? 1 : 0);
        s.evals += evaluated;
        double err[6], err3[6];
        rk_combine<M>(s, [&](int st, int i) { return K(P, st, i)[slot]; }, ynext, err, err3);
        for (int i = 0; i < 6; ++i) k0[i] = K(P, 0, i)[slot];
        int32_t code = -1;
        const int32_t d = attempt_decide<M>(A, s, k0, ynext, err, err3, &en, &code);
        if (P.bad[slot]) {
            traj_fail(A, s, traj, P.bad[slot] == 2 ? kWatchdog : P.bad[slot] == 3 ? kFrameTime : kGravityRadius);
        } else if (d == kFail) {
            traj_fail(A, s, traj, code);
        } else if (d == kAccept) {
            const double* dy_next = nullptr;
            if (T::FSAL) {
                for (int i = 0; i < 6; ++i) dyn[i] = K(P, T::S - 1, i)[slot];
                dy_next = dyn;
            } else if (dense && (s.flags & (kSegSampled | kEcl))) {
                for (int i = 0; i < 6; ++i) dyn[i] = K(P, T::S, i)[slot];
                dy_next = dyn;
                ++s.evals;  // counted on accept only, as the reference evaluates it
            }
            if (M != kDopri5Compat && (s.flags & kEcl)) {
                // most steps are certified free of crossings after a few
                // splits; the rest go to the warp
                if (ecl_accept_pre<M>(A, s, traj, ynext, k0, dyn, &tn, &req)) {
                    const EclGeo G{&A.force, s.jd0};
                    bool found = false;
                    EclBracket br{};
                    const int32_t e =
                        ecl_first_crossing(G, req.H, req.from, req.t1, &found, &br, kEclSoloSplits, &req.start);
                    if (e == kEclDefer) scan = true;
                    else ecl_accept_post<M>(A, s, traj, tn, ynext, k0, dyn, en, e, found, br);
                }
            } else
                attempt_accept<M>(A, s, traj, ynext, k0, dy_next, en);
        }
    }
    if (A.force.srp) {
        // the warp scans each waiting row's step together, one row at a time
        int32_t scan_err = kOk;
        bool scan_found = false;
        EclBracket scan_br{};
        unsigned want = __ballot_sync(0xffffffffu, scan);
        while (want) {
            const int leader = __ffs(want) - 1;
            want &= want - 1;
            EclPath H;
            for (int i = 0; i < 3; ++i) {
                H.p0[i] = __shfl_sync(0xffffffffu, req.H.p0[i], leader);
                H.v0[i] = __shfl_sync(0xffffffffu, req.H.v0[i], leader);
                H.p1[i] = __shfl_sync(0xffffffffu, req.H.p1[i], leader);
                H.v1[i] = __shfl_sync(0xffffffffu, req.H.v1[i], leader);
            }
            H.t0 = __shfl_sync(0xffffffffu, req.H.t0, leader);
            H.t1 = __shfl_sync(0xffffffffu, req.H.t1, leader);
            const double from = __shfl_sync(0xffffffffu, req.from, leader);
            const double t1 = __shfl_sync(0xffffffffu, req.t1, leader);
            const double jd0 = __shfl_sync(0xffffffffu, s.jd0, leader);
            EclPoint q;
            q.t = __shfl_sync(0xffffffffu, req.start.t, leader);
            for (int i = 0; i < 3; ++i) {
                q.p[i] = __shfl_sync(0xffffffffu, req.start.p[i], leader);
                q.v[i] = __shfl_sync(0xffffffffu, req.start.v[i], leader);
            }
            q.side = __shfl_sync(0xffffffffu, req.start.side, leader);
            q.margin = __shfl_sync(0xffffffffu, req.start.margin, leader);
            const EclGeo G{&A.force, jd0};
            bool found = false;
            EclBracket br{};
            const int32_t e = ecl_first_crossing_warp(G, H, from, t1, ecl_ws[threadIdx.x >> 5], &found, &br, &q);
            if (lane == leader) {
                scan_err = e;
                scan_found = found;
                scan_br = br;
            }
        }
        if (scan) ecl_accept_post<M>(A, s, traj, tn, ynext, k0, dyn, en, scan_err, scan_found, scan_br);
    }
    if (active) {
        if (s.phase == kNeedSegment) seg_begin<M>(A, s, traj);
        if (s.phase == kStepping) {
            const int32_t f = attempt_begin<M>(A, s, timed_out != 0);
            if (f >= 0) traj_fail(A, s, traj, f);
            else keep = true;
        }
        P.st[traj] = s;
    }
    append_active(P.idx[cur ^ 1], &P.count[cur ^ 1], traj, keep);  // whole warps take part in the ballot
}

// Rows still active when the host gives up (wall-clock watchdog).
template <int M>
__global__ void __launch_bounds__(kBlock) pl_abort(PropArgs A, PipeBufs P, int cur) {
    const int slot = blockIdx.x * blockDim.x + threadIdx.x;
    if (slot >= P.count[cur]) return;
    const int32_t traj = P.idx[cur][slot];
    TrajState s = P.st[traj];
    traj_fail(A, s, traj, kWatchdog);
    P.st[traj] = s;
}

// ------------------------------------------------------------------- host
// Stages whose instants are prepared at once: as many as leave their
// quantities (248 B a row and stage, 168 in the GMST frame) in L2 beside what
// the stages themselves touch, at least one.  The ring has one more, the
// stage before a group, which is finished after the group is prepared.
static int times_group(int64_t cap, int fields) {
    const int64_t one = cap * fields * 8;
    const int64_t g = one > 0 ? ((int64_t)96 << 20) / one : kStageBufs;
    return (int)(g < 1 ? 1 : (g > kStageBufs ? kStageBufs : g));
}

size_t pipeline_bytes(int64_t cap, int iau, int drag) {
    PipeBufs P{};
    pipeline_carve(P, nullptr, cap, iau, drag);
    return (size_t)(uintptr_t)P.dcount + 2 * (size_t)P.ring * sizeof(int32_t) + 256;
}

void pipeline_carve(PipeBufs& P, void* base, int64_t cap, int iau, int drag) {
    size_t off = 0;
    auto take = [&](size_t bytes) {
        off = (off + 255) & ~(size_t)255;
        char* p = (char*)base + off;
        off += bytes;
        return (void*)p;
    };
    const size_t c = (size_t)cap;
    P.cap = cap;
    P.st = (TrajState*)take(c * sizeof(TrajState));
    P.idx[0] = (int32_t*)take(c * 4);
    P.idx[1] = (int32_t*)take(c * 4);
    P.count = (int32_t*)take(2 * 4);
    P.k = (double*)take((size_t)kStageBufs * 6 * c * 8);
    P.sp = (double*)take(6 * c * 8);
    P.iau = iau;
    P.fields = kTimesFields + (iau ? kTimesIau : kTimesGmst) + (drag ? kTimesDrag : 0);
    P.ring = times_group(cap, P.fields) + 1;
    P.tq = (double*)take((size_t)P.ring * P.fields * c * 8);
    P.part = (double*)take(3 * c * 8);
    P.agrav = (double*)take(3 * c * 8);
    P.adrag = (double*)take(3 * c * 8);
    P.amcd = (double*)take(2 * c * 8);
    P.skip = (int32_t*)take(c * 4);
    P.bad = (int32_t*)take(c * 4);
    P.dlist[0] = (int32_t*)take(c * 4);
    P.dlist[1] = (int32_t*)take(c * 4);
    P.ef = (double*)take(3 * c * 8);
    P.agx = (double*)take(3 * c * 8);
    P.fall = (int32_t*)take(c * 4);
    P.flist = (int32_t*)take(c * 4);
    P.fcount = (int32_t*)take(4);
    P.dcount = (int32_t*)take(2 * (size_t)P.ring * 4);  // last: pipeline_bytes measures up to it
}

template <int M>
static cudaError_t run(const PropArgs& A, const PipeBufs& P, cudaStream_t user, double max_seconds,
                       int gthreads, int gslots, KernelTimes* times) {
    using T = Tab<M>;
    // the dense stage: the end-of-step derivative of sampled segments and of
    // the eclipse coordinator's Hermite scan
    const bool dense = (A.out_mode != kOutFinalEci || A.force.srp) && !T::FSAL;
    const int stages = T::S + (dense ? 1 : 0);
    // equal groups of at most P.ring - 1 stages
    const int groups = (stages + P.ring - 2) / (P.ring - 1), group = (stages + groups - 1) / groups;
    const int blocks = (int)((A.n + kBlock - 1) / kBlock);
    constexpr int kLanesHigh = BQP_DRAG_LANES_HIGH, kLanesLow = BQP_DRAG_LANES_LOW;
    const int dblocks_hi = (int)((A.n * kLanesHigh + kDragBlock - 1) / kDragBlock);
    const int dblocks_lo = (int)((A.n * kLanesLow + kDragBlock - 1) / kDragBlock);
    // more registers a thread while a stage's rows still fit in one wave
    auto dker = A.ordered ? pl_drag<kLanesHigh, kLanesLow, BQP_DRAG_MIN_BLOCKS_FEW, 3>
                : dblocks_hi <= 2 * device_sm_count() ? pl_drag<kLanesHigh, kLanesLow, BQP_DRAG_MIN_BLOCKS_FEW, 0>
                                                      : pl_drag<kLanesHigh, kLanesLow, BQP_DRAG_MIN_BLOCKS, 0>;
    const int cblocks = (int)((A.n + kDragBlock - 1) / kDragBlock);
    // with the surrogate, the exact stage covers only the degrees it leaves out
    const bool sur = A.sur.P != nullptr;
    const GravTable GT = sur ? A.sur.low : A.grav;
    // the surrogate's residual check also runs the whole exact field
    const bool check = sur && A.sur.check > 0.0;
    // with drag beside it, 128 threads (31 K registers an SM) leave the other
    // half of the registers to the drag kernel, and four warps of four rows a
    // lane still keep the FP64 pipe as busy as the table reads let it: 65,536
    // rows 331 ms a pass against 398 with 256 threads, 20,001 rows 179 and 210
    if (A.force.drag && !times && gthreads == 256 && !A.ordered) gthreads = 128;
    GravLaunch G = gravity_launch(GT, A.n, device_sm_count(), gthreads, gslots);
    GravLaunch GF = check ? gravity_launch(A.sur.full, A.n, device_sm_count(), gthreads, gslots) : G;
    auto gker = pl_gravity_of(G), gker_full = pl_gravity_of(GF);
    // the larger shared memory last: the two may be one kernel
    cudaError_t e = cudaSuccess;
    if (check && GF.smem < G.smem) e = gravity_ready(GF, gker_full);
    if (e == cudaSuccess) e = gravity_ready(G, gker);
    if (e == cudaSuccess && check && GF.smem >= G.smem) e = gravity_ready(GF, gker_full);
    if (e != cudaSuccess) return e;
    if (A.force.fit) {
        // the fixed-node fits: the same table for every context, ordered on
        // the caller's stream before this call's kernels
        if (!A.fit_host) return cudaErrorInvalidValue;
        e = cudaMemcpyToSymbolAsync(jb::c_fixed_fit, A.fit_host, sizeof(jb::JbFit), 0, cudaMemcpyHostToDevice, user);
        if (e != cudaSuccess) return e;
    }
    // one CTA per SM (the table fills shared memory)
    const int gctas = G.grid(A.n), gctas_full = GF.grid(A.n);

    // private stream ordered after the caller's stream (graphs need a
    // capturable stream)
    // and a second one, whose kernels give way to the first's: a stage's drag
    // runs beside its gravity (one after the other while kernels are timed)
    int prio_low = 0, prio_high = 0;
    cudaDeviceGetStreamPriorityRange(&prio_low, &prio_high);
    cudaStream_t st, st2;
    e = cudaStreamCreateWithPriority(&st, cudaStreamNonBlocking, prio_high);
    if (e != cudaSuccess) return e;
    e = cudaStreamCreateWithPriority(&st2, cudaStreamNonBlocking, prio_low);
    if (e != cudaSuccess) {
        cudaStreamDestroy(st);
        return e;
    }
    const bool beside = A.force.drag && A.force.gravity_on && !times;
    cudaEvent_t ev_in, ev_out, ev_cnt, ev_fork, ev_join;
    cudaEventCreateWithFlags(&ev_fork, cudaEventDisableTiming);
    cudaEventCreateWithFlags(&ev_join, cudaEventDisableTiming);
    cudaEventCreateWithFlags(&ev_in, cudaEventDisableTiming);
    cudaEventCreateWithFlags(&ev_out, cudaEventDisableTiming);
    cudaEventCreateWithFlags(&ev_cnt, cudaEventDisableTiming);
    cudaEventRecord(ev_in, user);
    cudaStreamWaitEvent(st, ev_in, 0);
    int32_t* h_count = nullptr;
    cudaMallocHost(&h_count, sizeof(int32_t));

    cudaMemsetAsync(P.count, 0, 2 * sizeof(int32_t), st);
    if (check) cudaMemsetAsync(P.fall, 0, (size_t)A.n * sizeof(int32_t), st);
    pl_init<M><<<blocks, kBlock, 0, st>>>(A, P);

    // instrumentation: an event-record node on each side of every timed
    // kernel of the graph; the host sums the durations after each replay
    std::vector<cudaEvent_t> evs;
    std::vector<int> ev_class;  // class of the kernel between evs[2i] and evs[2i+1]
    auto timed = [&](int cls, auto&& launch) {
        if (!times) {
            launch();
            return;
        }
        cudaEvent_t a, b;
        cudaEventCreate(&a);
        cudaEventCreate(&b);
        cudaEventRecordWithFlags(a, st, cudaEventRecordExternal);
        launch();
        cudaEventRecordWithFlags(b, st, cudaEventRecordExternal);
        evs.push_back(a);
        evs.push_back(b);
        ev_class.push_back(cls);
    };
    // one graph = two attempts (active list 0 -> 1 -> 0)
    auto enqueue_attempt = [&](int cur, int timed_out) {
        for (int s = 0; s < stages; ++s) {
            timed(kKcPrep, [&] {
                if (s % group == 0)
                    pl_times<M><<<dim3(blocks, std::min(group, stages - s)), kBlock, 0, st>>>(A, P, cur, s);
                pl_prep<M><<<blocks, kBlock, 0, st>>>(A, P, cur, s);
            });
            cudaStream_t sd = st;
            if (beside) {
                sd = st2;
                cudaEventRecord(ev_fork, st);
                cudaStreamWaitEvent(st2, ev_fork, 0);
            }
            if (A.force.gravity_on)
                timed(kKcGravity, [&] {
                    gravity_run(G, gker, gctas, st, GT, G.aux, P, cur, s, P.agrav, nullptr, nullptr);
                    if (sur) {
                        pl_earth_fixed<<<blocks, kBlock, 0, st>>>(P, cur, s);
                        launch_surrogate_stage(A.sur, &P.count[cur], A.n, P.ef, P.agrav, 1, P.cap, st);
                        if (check && s == 0) {
                            // the exact field of every evaluated row, then the verdicts
                            cudaMemsetAsync(P.fcount, 0, sizeof(int32_t), st);
                            gravity_run(GF, gker_full, gctas_full, st, A.sur.full, GF.aux, P, cur, s, P.agx, nullptr,
                                        nullptr);
                            pl_sur_check<<<blocks, kBlock, 0, st>>>(P, cur, A.sur.check);
                        } else if (check) {
                            // the rows on the exact field for this step
                            gravity_run(GF, gker_full, gctas_full, st, A.sur.full, GF.aux, P, cur, s, P.agrav, P.flist,
                                        P.fcount);
                        }
                    }
                });
            if (A.force.drag)
                timed(kKcDrag, [&] {
                    if (A.force.atm_model == 4)
                        dker<<<dblocks_hi + dblocks_lo, kDragBlock, 0, sd>>>(A.force, P, s, dblocks_hi);
                    else if (A.force.drag_fp32)
                        pl_drag_coarse<2><<<2 * cblocks, kDragBlock, 0, sd>>>(A.force, P, s, cblocks);
                    else
                        pl_drag_coarse<1><<<2 * cblocks, kDragBlock, 0, sd>>>(A.force, P, s, cblocks);
                });
            if (beside) {
                cudaEventRecord(ev_join, st2);
                cudaStreamWaitEvent(st, ev_join, 0);
            }
        }
        timed(kKcControl, [&] { pl_control<M><<<blocks, kBlock, 0, st>>>(A, P, cur, dense ? 1 : 0, timed_out); });
    };
    auto collect = [&]() {
        for (size_t i = 0; i < ev_class.size(); ++i) {
            float ms = 0.0f;
            if (cudaEventElapsedTime(&ms, evs[2 * i], evs[2 * i + 1]) == cudaSuccess) {
                times->ms[ev_class[i]] += ms;
                times->launches[ev_class[i]] += 1;
            }
        }
    };
    cudaGraph_t graph = nullptr;
    cudaGraphExec_t exec = nullptr;
    e = cudaStreamBeginCapture(st, cudaStreamCaptureModeThreadLocal);
    if (e == cudaSuccess) {
        enqueue_attempt(0, 0);
        enqueue_attempt(1, 0);
        e = cudaStreamEndCapture(st, &graph);
    }
    if (e == cudaSuccess) e = cudaGraphInstantiate(&exec, graph, 0);
    const auto t_start = std::chrono::steady_clock::now();
    // host loop: replay, keep one replay in flight ahead of the count check
    int64_t replays = 0;
    bool done = false;
    while (e == cudaSuccess && !done) {
        e = cudaGraphLaunch(exec, st);
        if (e != cudaSuccess) break;
        cudaMemcpyAsync(h_count, &P.count[0], sizeof(int32_t), cudaMemcpyDeviceToHost, st);
        cudaEventRecord(ev_cnt, st);
        if (times) {
            // no replay in flight while the events of this one are read
            e = cudaEventSynchronize(ev_cnt);
            if (e != cudaSuccess) break;
            collect();
        }
        e = cudaGraphLaunch(exec, st);  // speculative: cheap when nothing is active
        if (e != cudaSuccess) break;
        e = cudaEventSynchronize(ev_cnt);
        if (times && e == cudaSuccess) {
            e = cudaStreamSynchronize(st);
            if (e == cudaSuccess) collect();
        }
        replays += 2;
        if (*h_count == 0) done = true;
        const double elapsed =
            std::chrono::duration<double>(std::chrono::steady_clock::now() - t_start).count();
        if (!done && max_seconds > 0.0 && elapsed > max_seconds) {
            cudaStreamSynchronize(st);
            pl_abort<M><<<blocks, kBlock, 0, st>>>(A, P, 0);
            done = true;
        }
    }
    if (e == cudaSuccess) e = cudaGetLastError();
    cudaEventRecord(ev_out, st);
    cudaStreamWaitEvent(user, ev_out, 0);
    cudaStreamSynchronize(st);
    if (exec) cudaGraphExecDestroy(exec);
    if (graph) cudaGraphDestroy(graph);
    cudaFreeHost(h_count);
    for (cudaEvent_t ev : evs) cudaEventDestroy(ev);
    cudaEventDestroy(ev_in);
    cudaEventDestroy(ev_out);
    cudaEventDestroy(ev_cnt);
    cudaEventDestroy(ev_fork);
    cudaEventDestroy(ev_join);
    cudaStreamDestroy(st2);
    cudaStreamDestroy(st);
    return e;
}

cudaError_t launch_pipeline(const PropArgs& A, const PipeBufs& P, int method, cudaStream_t st, double max_seconds,
                            int gravity_threads, int gravity_slots, KernelTimes* times) {
    if (A.n <= 0) return cudaSuccess;
    if (gravity_threads <= 0) gravity_threads = 256;
    switch (method) {
        case kDopri5: return run<kDopri5>(A, P, st, max_seconds, gravity_threads, gravity_slots, times);
        case kDop853: return run<kDop853>(A, P, st, max_seconds, gravity_threads, gravity_slots, times);
        case kDopri5Compat:
            return run<kDopri5Compat>(A, P, st, max_seconds, gravity_threads, gravity_slots, times);
        case kVern7: return run<kVern7>(A, P, st, max_seconds, gravity_threads, gravity_slots, times);
        case kVern9: return run<kVern9>(A, P, st, max_seconds, gravity_threads, gravity_slots, times);
        default: return cudaErrorInvalidValue;
    }
}

}  // namespace bqp
