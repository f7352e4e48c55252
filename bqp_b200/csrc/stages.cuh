// What a row goes through in one step attempt, stage by stage, shared by the
// stage kernels (pipeline.cu: one kernel per part over all rows) and the
// attempt kernel (attempt.cu: all parts in one kernel, a few rows per CTA).
#pragma once
#include "kernels.cuh"
#include "launch.h"
#include "traj.cuh"

namespace bqp {

constexpr int kBlock = 256;
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

// ------------------------------------------------------------------ instants
// Stage `st` (at time ts) of one row: the parts in `tasks`, each independent of
// the others' output.
//
// Everything here is known when the attempt begins, so the stages' long FP64
// chains (the Kepler solve, the Sun and Moon series, the frame) run side by
// side once an attempt instead of one after the other before each stage's
// force.
enum TimesTask : int { kTimesOrbit = 1, kTimesFrame = 2, kTimesSun = 4, kTimesMoon = 8, kTimesAll = 15 };
__device__ __forceinline__ void times_row(const PropArgs& A, const PipeBufs& P, const TrajState& s, int slot, int st,
                                          double ts, int tasks) {
    const StageTimes Q(P, st);
    const ForceParams& fp = A.force;
    if (tasks & kTimesOrbit) {
        double rs[6];
        baseline_state(baseline_new(s.cur), ts - s.ct0, rs);
        for (int i = 0; i < 6; ++i) Q.baseline(i, slot) = rs[i];
    }
    const double jd = utc_jd_at(s.jd0, ts);
    const bool sun_on = fp.sun || (fp.drag && s.cd != 0.0 && s.am != 0.0) || s.side >= 0;
    // the Earth-fixed frame, for itself and for the Sun's place in it
    double r[12];
    if (tasks & kTimesFrame || (tasks & kTimesSun && sun_on && fp.drag)) {
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
            for (int e = 0; e < 9; ++e) r[e] = F.r[e];
            for (int e = 0; e < 3; ++e) r[9 + e] = F.w[e];
        } else {
            r[0] = 0.0;
            r[1] = 1.0;
            if (fp.gravity_on || fp.drag) sincos(gmst_rad(jd), &r[0], &r[1]);
        }
    }
    if (tasks & kTimesFrame) {
        Q.jd(slot) = jd;
        for (int e = 0; e < (P.iau ? kTimesIau : kTimesGmst); ++e) Q.frame(e, slot) = r[e];
    }
    if (tasks & kTimesSun && sun_on) {
        double sun[3];
        sun_at(fp.eph_sun, jd, sun);
        for (int i = 0; i < 3; ++i) Q.sun(i, slot) = sun[i];
        if (fp.drag) {
            // JB2008 adapter (rhs.rs:3551-3776), as Encke::density_at: the
            // Sun's side of it
            double si[3];
            if (P.iau) {
                ft::to_itrs(r, sun, si);
            } else {
                si[0] = fma(r[1], sun[0], r[0] * sun[1]);
                si[1] = fma(-r[0], sun[0], r[1] * sun[1]);
                si[2] = sun[2];
            }
            const double sun_r = sqrt(fma(si[0], si[0], fma(si[1], si[1], si[2] * si[2])));
            Q.drag(P, 0, slot) = si[0];
            Q.drag(P, 1, slot) = si[1];
            Q.drag(P, 2, slot) = asin(fmin(1.0, fmax(-1.0, si[2] / sun_r)));
        }
    }
    if (tasks & kTimesMoon) {
        if (fp.moon) {
            double moon[3];
            moon_at(fp.eph_moon, jd, moon);
            for (int i = 0; i < 3; ++i) Q.moon(i, slot) = moon[i];
        }
        if (fp.drag && sun_on) {
            // and the drivers'
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
}

// Stage st's time in row s.  st == S is the dense-output stage of the sampled
// non-FSAL path: f(t_next, y_next) evaluated before the controller decides
// (the reference evaluates it after an accept).
template <int M>
__device__ __forceinline__ double stage_time(const TrajState& s, int st) {
    return st < Tab<M>::S ? fma(Tab<M>::c(st), s.hs, s.t) : next_time(s);
}

// --------------------------------------------------------------- preparation
struct Vec3 {
    double x, y, z;
};
// SRP (on the leg's fixed side), third bodies and Battin's term at sp, the
// baseline's rs plus the deviation yt.  Out of line: which neighbouring
// products and sums the compiler fuses depends on what it compiles together,
// and PropArgs::ordered rows take the same bits in both engines' kernels.
static __device__ __noinline__ Vec3 stage_accel(const ForceParams& fp, Vec3 p, Vec3 sun_v, Vec3 moon_v, Vec3 base,
                                                Vec3 dev, double r2, double am, int side) {
    const double sp[3] = {p.x, p.y, p.z}, sun[3] = {sun_v.x, sun_v.y, sun_v.z},
                 moon[3] = {moon_v.x, moon_v.y, moon_v.z}, rs[3] = {base.x, base.y, base.z},
                 yt[3] = {dev.x, dev.y, dev.z};
    double acc[3] = {0.0, 0.0, 0.0};
    if (side >= 0) srp_accel(sp, sun, fp.p_sun, fp.cr, am, side, acc);
    if (fp.sun) third_body(sp, sun, fp.mu_sun, acc);
    if (fp.moon) third_body(sp, moon, fp.mu_moon, acc);
    battin(rs, yt, r2, sqrt(r2), acc);
    return {acc[0], acc[1], acc[2]};
}

// Stage st of one row: its state y_s, the perturbed state, third body, Battin;
// the stage before it is finished.  False where the first stage is taken over
// from the step before; *r2 is the squared radius (drag).
template <int M>
__device__ __forceinline__ bool prep_row(const PropArgs& A, const PipeBufs& P, const TrajState& s, int slot, int st,
                                         double* r2_out) {
    using T = Tab<M>;
    if (st == 0) {
        P.bad[slot] = 0;
        if (s.flags & kHaveK1) {
            for (int i = 0; i < 6; ++i) K(P, 0, i)[slot] = s.k1c[i];
            P.skip[slot] = 1;
            return false;
        }
    } else if (!(st == 1 && P.skip[slot])) {
        finish_stage(P, st - 1, slot);
    }
    P.skip[slot] = 0;
    // stage state
    double yt[6];
    for (int i = 0; i < 6; ++i) yt[i] = s.y[i];
    if (st < T::S) {
#pragma unroll
        for (int j = 0; j < T::S; ++j) {
            if (j >= st) break;
            const double a = s.hs * T::a(st, j);
            if (a != 0.0)
                for (int i = 0; i < 6; ++i) yt[i] = fma(K(P, j, i)[slot], a, yt[i]);
        }
    } else {
        // y_next exactly as rk_combine forms it
#pragma unroll
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
    const bool need_sun = fp.sun || (fp.drag && s.cd != 0.0 && s.am != 0.0) || s.side >= 0;
    Vec3 sun{}, moon{};
    if (need_sun) sun = {Q.sun(0, slot), Q.sun(1, slot), Q.sun(2, slot)};
    if (fp.moon) moon = {Q.moon(0, slot), Q.moon(1, slot), Q.moon(2, slot)};
    const double r2 = fma(sp[0], sp[0], fma(sp[1], sp[1], sp[2] * sp[2]));
    const Vec3 part = stage_accel(fp, {sp[0], sp[1], sp[2]}, sun, moon, {rs[0], rs[1], rs[2]}, {yt[0], yt[1], yt[2]}, r2,
                                  s.am, s.side);
    const double acc[3] = {part.x, part.y, part.z};
    for (int i = 0; i < 3; ++i) P.part[(size_t)i * P.cap + slot] = acc[i];
    if (fp.drag) {
        P.amcd[slot] = s.am;
        P.amcd[P.cap + slot] = s.cd;
    } else {
        for (int i = 0; i < 3; ++i) P.adrag[(size_t)i * P.cap + slot] = 0.0;
    }
    if (!fp.gravity_on)
        for (int i = 0; i < 3; ++i) P.agrav[(size_t)i * P.cap + slot] = 0.0;
    *r2_out = r2;
    return true;
}

// ---------------------------------------------------------------------- drag
// One state per group of L lanes (jb::density_group; q: the lane in its group,
// gmask the group's lanes): the JB2008 model is the longest serial chain of the
// force call, and it is bound by that latency, not by throughput.
// kForm 0: the exact model; 1, 2: the coarse profiles in FP64 and in FP32; 3:
// the exact model in the order of PropArgs::ordered; 4: the coarse profiles in
// FP64 by four lanes.
template <int L, int kForm>
__device__ __forceinline__ void drag_row(const ForceParams& fp, const PipeBufs& P, int st, int slot, int q,
                                         unsigned gmask) {
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
            const double hy = fma(pi[1], si0, -(pi[0] * si1)), hx = fma(pi[0], si0, pi[1] * si1);
            double ha, lat;
            if (kForm == 4) {
                // both angles in one call, on lanes 0 and 1
                const double v = atan2(q & 1 ? pi[2] : hy, q & 1 ? sqrt(fma(pi[0], pi[0], pi[1] * pi[1])) : hx);
                ha = __shfl_sync(gmask, v, 0, 4);
                lat = __shfl_sync(gmask, v, 1, 4);
            } else {
                ha = atan2(hy, hx);
                lat = asin(fmin(1.0, fmax(-1.0, pi[2] / sat_r)));
            }
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
            else if (kForm == 4)
                rho = jb::density_coarse_quad(E, dec, ha, lat, alt_m, dr, fp.atm_model, &fp.plan, q, gmask);
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

// ------------------------------------------------------------------- control
// Splits a row's own thread may take on its crossing scan before the warp
// takes it over.
#ifndef BQP_ECL_SOLO_SPLITS
#define BQP_ECL_SOLO_SPLITS 4
#endif
constexpr int64_t kEclSoloSplits = BQP_ECL_SOLO_SPLITS;

// The end of an attempt for the 32 rows of a warp (all lanes take part; row
// `traj` in slot `slot` where active): the last stage, the error, accept or reject,
// samples, rectification, the next attempt; rows that go on are appended to
// `next`.  ws: the warp's store for the cooperative eclipse scan (SRP rows).
template <int M>
__device__ __forceinline__ void control_warp(const PropArgs& A, const PipeBufs& P, int32_t traj, int slot,
                                             bool active, int32_t* next, int32_t* next_count, EclWarpStore& ws,
                                             int dense) {
    using T = Tab<M>;
    const int lane = threadIdx.x & 31;
    bool keep = false;
    TrajState s;
    bool scan = false;  // an accepted SRP step waiting for its crossing scan
    EclScanReq req;
    double tn = 0.0, en = 0.0, ynext[6], k0[6], dyn[6];
    if (active) {
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
            const int32_t e = ecl_first_crossing_warp(G, H, from, t1, ws, &found, &br, &q);
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
            const int32_t f = attempt_begin<M>(A, s, false);
            if (f >= 0) traj_fail(A, s, traj, f);
            else keep = true;
        }
        P.st[traj] = s;
    }
    append_active(next, next_count, traj, keep);  // whole warps take part in the ballot
}

// Whether the call's wall-clock limit is over, by the device's clock.
__device__ __forceinline__ bool over_time(const PropArgs& A, const PipeBufs& P) {
    return A.ctrl.max_kernel_ns > 0 && (int64_t)(global_ns() - *P.started) > A.ctrl.max_kernel_ns;
}

// --------------------------------------------------------------------- init
template <int M>
__global__ void __launch_bounds__(kBlock) pl_init(const __grid_constant__ PropArgs A, const __grid_constant__ PipeBufs P) {
    const int64_t traj = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    bool keep = false;
    if (traj == 0) {
        *P.started = global_ns();
        P.over[0] = P.over[1] = 0;
    }
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

// Rows still active when the host gives up (wall-clock watchdog).
template <int M>
__global__ void __launch_bounds__(kBlock) pl_abort(const __grid_constant__ PropArgs A, const __grid_constant__ PipeBufs P,
                                                   int cur) {
    const int slot = blockIdx.x * blockDim.x + threadIdx.x;
    if (slot >= P.count[cur]) return;
    const int32_t traj = P.idx[cur][slot];
    TrajState s = P.st[traj];
    traj_fail(A, s, traj, kWatchdog);
    P.st[traj] = s;
}

}  // namespace bqp
