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
#include <cstdint>
#include <vector>

#include "replay.h"
#include "stages.cuh"

namespace bqp {

namespace {

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
}  // namespace

// -------------------------------------------------------------------- times
// Stages st0 .. st0 + gridDim.y - 1 of the current attempt, one stage of one
// row a thread.  With 65,536 rows at 70x70 the stage kernels' preparation
// went from 22.8 to 20.5 us a stage, with 200 rows from 21 to 14.5.
template <int M>
__global__ void __launch_bounds__(kBlock) pl_times(const __grid_constant__ PropArgs A,
                                                   const __grid_constant__ PipeBufs P, int list, int counter, int st0) {
    const int slot = blockIdx.x * blockDim.x + threadIdx.x, st = st0 + blockIdx.y;
    if (blockIdx.x == 0 && threadIdx.x < 2) P.dcount[2 * (st % P.ring) + threadIdx.x] = 0;
    if (slot >= P.count[counter]) return;
    const TrajState& s = P.st[P.idx[list][slot]];
    if (st == 0 && (s.flags & kHaveK1)) return;
    times_row(A, P, s, slot, st, stage_time<M>(s, st), kTimesAll);
}

void launch_times(const PropArgs& A, const PipeBufs& P, int method, int list, int counter, int stages,
                  cudaStream_t st) {
    const dim3 grid((unsigned)((A.n + kBlock - 1) / kBlock), (unsigned)stages);
    switch (method) {
        case kDopri5: pl_times<kDopri5><<<grid, kBlock, 0, st>>>(A, P, list, counter, 0); break;
        case kDop853: pl_times<kDop853><<<grid, kBlock, 0, st>>>(A, P, list, counter, 0); break;
        case kDopri5Compat: pl_times<kDopri5Compat><<<grid, kBlock, 0, st>>>(A, P, list, counter, 0); break;
        case kVern7: pl_times<kVern7><<<grid, kBlock, 0, st>>>(A, P, list, counter, 0); break;
        case kVern9: pl_times<kVern9><<<grid, kBlock, 0, st>>>(A, P, list, counter, 0); break;
    }
}

// --------------------------------------------------------------------- prep
template <int M>
__global__ void __launch_bounds__(kBlock) pl_prep(const __grid_constant__ PropArgs A,
                                                  const __grid_constant__ PipeBufs P, int cur, int st) {
    const int slot = blockIdx.x * blockDim.x + threadIdx.x;
    if (st == 0 && blockIdx.x == 0 && threadIdx.x == 0) P.count[cur ^ 1] = 0;
    if (slot >= P.count[cur]) return;
    double r2;
    if (!prep_row<M>(A, P, P.st[P.idx[cur][slot]], slot, st, &r2) || !A.force.drag) return;
    // drag work list: states above ~510 km take the sweep fits (cheap),
    // the rest walk the quadrature; homogeneous warps in each list
    const int cls = sqrt(r2) - A.force.earth_radius >= 510.0 ? 0 : 1;
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
// Both drag lists go in one launch (blocks [0, nb_hi) take list 0 with LH
// lanes per state, the rest list 1 with LL), so that a stage's states are
// resident together in as few waves as the register budget allows.
template <int L, int kForm = 0>
__device__ __forceinline__ void drag_rows(const ForceParams& fp, const PipeBufs& P, int st, int list, int block) {
    const int gt = block * blockDim.x + threadIdx.x;
    const int item = gt / L;
    if (item >= P.dcount[2 * (st % P.ring) + list]) return;  // uniform across the group
    drag_row<L, kForm>(fp, P, st, P.dlist[list][item], gt % L, ((1u << L) - 1u) << ((threadIdx.x & 31) & ~(L - 1)));
}

template <int LH, int LL, int kMinBlocks, int kForm>
__global__ void __launch_bounds__(kDragBlock, kMinBlocks) pl_drag(const __grid_constant__ ForceParams fp,
                                                              const __grid_constant__ PipeBufs P, int st, int nb_hi) {
    if ((int)blockIdx.x < nb_hi) drag_rows<LH, kForm>(fp, P, st, 0, blockIdx.x);
    else drag_rows<LL, kForm>(fp, P, st, 1, blockIdx.x - nb_hi);
}

// The coarse profiles (atm_model 5-7), both altitude lists in one launch: above
// ~510 km a short chain per state on one lane; below, up to twelve panels one
// after the other, so four lanes take a state there (a node of each panel a
// lane).  20,001 rows, model 7: 152,141 us a pass, 178,363 with one lane in
// both.
#ifndef BQP_COARSE_MIN_BLOCKS
#define BQP_COARSE_MIN_BLOCKS 4
#endif
template <int LL, int kForm, int kFormLow>
__global__ void __launch_bounds__(kDragBlock, BQP_COARSE_MIN_BLOCKS)
    pl_drag_coarse(const __grid_constant__ ForceParams fp, const __grid_constant__ PipeBufs P, int st, int nb_hi) {
    if ((int)blockIdx.x < nb_hi) drag_rows<1, kForm>(fp, P, st, 0, blockIdx.x);
    else drag_rows<LL, kFormLow>(fp, P, st, 1, blockIdx.x - nb_hi);
}

// ------------------------------------------------------------------ control
template <int M>
__global__ void __launch_bounds__(kBlock) pl_control(const __grid_constant__ PropArgs A,
                                                     const __grid_constant__ PipeBufs P, int cur, int dense) {
    __shared__ EclWarpStore ecl_ws[kBlock / 32];
    const int slot = blockIdx.x * blockDim.x + threadIdx.x;
    const int count = P.count[cur];
    if (slot - (int)(threadIdx.x & 31) >= count) return;  // the whole warp is idle
    control_warp<M>(A, P, slot < count ? P.idx[cur][slot] : 0, slot, slot < count, P.idx[cur ^ 1], &P.count[cur ^ 1],
                    ecl_ws[threadIdx.x >> 5], dense);
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
    P.count = (int32_t*)take(3 * 4);
    P.started = (uint64_t*)take(8);
    P.over = (int32_t*)take(2 * 4);
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

cudaError_t ReplayRes::ready() {
    if (h_count) return cudaSuccess;
    int low = 0, high = 0;
    cudaDeviceGetStreamPriorityRange(&low, &high);
    cudaError_t e = cudaStreamCreateWithPriority(&st, cudaStreamNonBlocking, high);
    if (e == cudaSuccess) e = cudaStreamCreateWithPriority(&st2, cudaStreamNonBlocking, low);
    for (cudaEvent_t* ev : {&ev_in, &ev_out, &ev_cnt, &ev_order})
        if (e == cudaSuccess) e = cudaEventCreateWithFlags(ev, cudaEventDisableTiming);
    if (e == cudaSuccess) e = cudaMallocHost(&h_count, sizeof(int32_t));
    if (e != cudaSuccess) release();
    return e;
}

void ReplayRes::release() {
    if (h_count) cudaFreeHost(h_count);
    for (cudaEvent_t ev : {ev_in, ev_out, ev_cnt, ev_order})
        if (ev) cudaEventDestroy(ev);
    if (st2) cudaStreamDestroy(st2);
    if (st) cudaStreamDestroy(st);
    *this = ReplayRes{};
}

template <int M>
static cudaError_t run(const PropArgs& A, const PipeBufs& P, ReplayRes& R, cudaStream_t user, double max_seconds,
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
    cudaError_t e = gravity_ready(G, gker);
    if (e == cudaSuccess && check) e = gravity_ready(GF, gker_full);
    if (e != cudaSuccess) return e;
    e = upload_fixed_fit(A, user);
    if (e != cudaSuccess) return e;
    // one CTA per SM (the table fills shared memory)
    const int gctas = G.grid(A.n), gctas_full = GF.grid(A.n);

    const bool beside = A.force.drag && A.force.gravity_on && !times;
    // instrumentation: an event-record node on each side of every timed
    // kernel of the graph; the host sums the durations after each replay
    std::vector<cudaEvent_t> evs;
    std::vector<int> ev_class;  // class of the kernel between evs[2i] and evs[2i+1]
    auto timed = [&](cudaStream_t st, int cls, auto&& launch) {
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
    auto enqueue_attempt = [&](cudaStream_t st, cudaStream_t st2, const StreamOrder& order_after, int cur) {
        for (int s = 0; s < stages; ++s) {
            timed(st, kKcPrep, [&] {
                if (s % group == 0)
                    pl_times<M><<<dim3(blocks, std::min(group, stages - s)), kBlock, 0, st>>>(A, P, cur, cur, s);
                pl_prep<M><<<blocks, kBlock, 0, st>>>(A, P, cur, s);
            });
            cudaStream_t sd = st;
            if (beside) {
                sd = st2;
                order_after(st, st2);
            }
            if (A.force.gravity_on)
                timed(st, kKcGravity, [&] {
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
                timed(st, kKcDrag, [&] {
                    if (A.force.atm_model == 4)
                        dker<<<dblocks_hi + dblocks_lo, kDragBlock, 0, sd>>>(A.force, P, s, dblocks_hi);
                    else if (A.force.drag_fp32)
                        pl_drag_coarse<1, 2, 2><<<2 * cblocks, kDragBlock, 0, sd>>>(A.force, P, s, cblocks);
                    else if (A.ordered)
                        pl_drag_coarse<1, 1, 1><<<2 * cblocks, kDragBlock, 0, sd>>>(A.force, P, s, cblocks);
                    else
                        pl_drag_coarse<4, 1, 4><<<5 * cblocks, kDragBlock, 0, sd>>>(A.force, P, s, cblocks);
                });
            if (beside) {
                order_after(st2, st);
            }
        }
        timed(st, kKcControl, [&] { pl_control<M><<<blocks, kBlock, 0, st>>>(A, P, cur, dense ? 1 : 0); });
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
    e = replay(
        P, R, user, max_seconds, true, times != nullptr,
        [&](cudaStream_t st) {
            if (check) cudaMemsetAsync(P.fall, 0, (size_t)A.n * sizeof(int32_t), st);
            pl_init<M><<<blocks, kBlock, 0, st>>>(A, P);
        },
        [&](cudaStream_t st, cudaStream_t st2, const StreamOrder& order_after) {
            // one graph = two attempts (active list 0 -> 1 -> 0)
            enqueue_attempt(st, st2, order_after, 0);
            enqueue_attempt(st, st2, order_after, 1);
        },
        [&](cudaStream_t st) { pl_abort<M><<<blocks, kBlock, 0, st>>>(A, P, 0); }, collect);
    for (cudaEvent_t ev : evs) cudaEventDestroy(ev);
    return e;
}

cudaError_t launch_pipeline(const PropArgs& A, const PipeBufs& P, ReplayRes& R, int method, cudaStream_t st,
                            double max_seconds,
                            int gravity_threads, int gravity_slots, KernelTimes* times) {
    if (A.n <= 0) return cudaSuccess;
    if (gravity_threads <= 0) gravity_threads = 256;
    if (!times && gravity_threads == 256 && gravity_slots != 1 && gravity_slots != 2 && attempt_fits(A))
        return launch_attempts(A, P, R, method, st, max_seconds);
    switch (method) {
        case kDopri5: return run<kDopri5>(A, P, R, st, max_seconds, gravity_threads, gravity_slots, times);
        case kDop853: return run<kDop853>(A, P, R, st, max_seconds, gravity_threads, gravity_slots, times);
        case kDopri5Compat:
            return run<kDopri5Compat>(A, P, R, st, max_seconds, gravity_threads, gravity_slots, times);
        case kVern7: return run<kVern7>(A, P, R, st, max_seconds, gravity_threads, gravity_slots, times);
        case kVern9: return run<kVern9>(A, P, R, st, max_seconds, gravity_threads, gravity_slots, times);
        default: return cudaErrorInvalidValue;
    }
}

}  // namespace bqp
