// Attempt kernel: whole step attempts of a small batch in one launch.
//
// With a few thousand rows the stage kernels (pipeline.cu) are bound by what
// each costs whatever its rows: a launch and its gap, the staging of the field
// table, and one row's serial chain, three kernels a stage one after the other.
// Trajectories do not depend on one another, so here a CTA keeps a few rows
// (at most kAttemptRows) through all stages of its attempts: the instants'
// chains of all stages run side by side first (one part of one stage of one
// row a thread), then stage by stage a thread a row prepares, and four warps
// evaluate the drag (four or two lanes a row) while the others share the field's
// columns; the controller closes the attempt.  The table is staged once a
// launch, under the first attempt's instants.  The field's sums are added in the order
// of the shares, the same for every batch.
//
// us a pass, stage kernels -> attempt kernel: one satellite over an hour, every
// default 26,527 -> 14,435; 200 rows over 5,400 s 37,658 -> 25,269; 1,024 rows
// over a day on a 60 s grid 519,986 -> 249,360; 6,000 mixed rows 371,461 ->
// 286,615; 1,500 rows with SRP 261,000 -> 173,479.
//
// Its limit of 64 rows a CTA is what its arrays hold.  There (9,472 rows, 600 s,
// DOP853 at 1e-10, attempt kernel against stage kernels): 20x20 without drag
// 4,458 us and 7,334, 70x70 without drag 12,974 and 15,960, 70x70 with the fitted
// density 22,262 and 23,070, with the exact one 44,045 and 37,732; with SRP
// 157,266 and 207,844 (3,000 s).  Only the exact density at 70x70 runs
// slower here, from about 30 rows a CTA (32,411 and 30,860); it is 1.22 times
// as fast at 16.
#include <cuda_runtime.h>

#include <cstdint>

#include "gravity_cta.cuh"
#include "replay.h"
#include "stages.cuh"

namespace bqp {

namespace {

// 12 warps: 168 registers a thread, 4 warps for the drag, 8 (12 without drag)
// shares of the field's columns.
constexpr int kAttemptThreads = 384, kDragWarps = 4;
// rows a CTA keeps: two tiles of a warp, the controller's two warps
constexpr int kAttemptRows = 64;
// Attempts a CTA makes on its rows before the rows that go on are dealt out
// again.  CTAs then wait for one another once a launch, not once an attempt:
// with SRP a row that crosses the shadow's edge keeps its CTA's controller for
// most of a millisecond, a few rows of 1,500 in every attempt.
constexpr int kAttemptRounds = 16;
// Rows a CTA up to which the exact density takes four lanes a row, two beyond.
// Up to 25 rows four fit in one pass of the drag's warps whatever share of them
// is above ~510 km; 32 to 64 rows take 4 to 7 % less with two (64 rows, 20x20,
// 600 s: 30,276 us against 32,288).  The forms do not give the same bits, so
// the rows a CTA are the launch's, not a CTA's own: which rows share a CTA, and
// how many of them are above, differs from run to run.  The coarse profiles
// take four lanes at any count (48 rows a CTA, 20x20: 13,246 us; 14,395 with
// one lane a row where four did not fit in one pass).
constexpr int kFourLanesRows = 25;

// the table and the shares' sums, beside the static arrays (at_attempt's)
constexpr size_t kAttemptStatic = 12 * 1024, kAttemptSmem = kSmemLimit - kAttemptStatic;
static_assert(sizeof(uint64_t) + kAttemptRows / 32 * sizeof(EclWarpStore) + (4 * kAttemptRows + 8) * sizeof(int32_t) + 64 <=
              kAttemptStatic);
size_t attempt_smem_bytes(const GravTable& T, int shares) {
    return ((size_t)shares * 3 * kAttemptRows + kGravityTabPad) * sizeof(double) + T.bytes;
}

// Drag of the CTA's rows by its first warps, L lanes a row; the rows of one
// list (above / below ~510 km, homogeneous code paths) to a warp.
template <int L, int kForm>
__device__ __noinline__ void attempt_drag(const ForceParams& fp, const PipeBufs& P, int st, int b0,
                                          const int32_t* rows_hi, int n_hi, const int32_t* rows_lo, int n_lo) {
    constexpr int kGroups = 32 / L;
    const int lane = threadIdx.x & 31, g = lane / L, q = lane % L;
    const unsigned gmask = (L == 32 ? 0xffffffffu : ((1u << L) - 1u)) << (lane & ~(L - 1));
    const int warps_hi = (n_hi + kGroups - 1) / kGroups, warps_lo = (n_lo + kGroups - 1) / kGroups;
    for (int u = threadIdx.x >> 5; u < warps_hi + warps_lo; u += kDragWarps) {
        const bool hi = u < warps_hi;
        const int i = (hi ? u : u - warps_hi) * kGroups + g;
        if (i < (hi ? n_hi : n_lo)) drag_row<L, kForm>(fp, P, st, b0 + (hi ? rows_hi[i] : rows_lo[i]), q, gmask);
    }
}

// Earth-fixed position of row r of the CTA in stage st; left as it is (a valid
// dummy) for rows that need no force.  False where the field is NaN: an
// invalid radius, or the table copy was lost (`marks`: and record it).
__device__ __forceinline__ bool attempt_position(const PipeBufs& P, int st, int b0, int rows, int r, bool marks,
                                                 bool staged, double* x, double* y, double* z) {
    const int sl = b0 + r;
    if (r >= rows || P.skip[sl]) return staged;
    if (!staged) {
        if (marks) P.bad[sl] = 2;
        return false;
    }
    const double e[3] = {P.sp[sl], P.sp[P.cap + sl], P.sp[2 * P.cap + sl]};
    double f[3];
    slot_to_itrs(P, StageTimes(P, st), sl, e, f);
    const double r2 = fma(f[0], f[0], fma(f[1], f[1], f[2] * f[2]));
    if (!(isfinite(r2) && r2 > 0.0)) {
        if (marks && !P.bad[sl]) P.bad[sl] = 1;
        return false;
    }
    *x = f[0];
    *y = f[1];
    *z = f[2];
    return true;
}

// Share w of the field at the CTA's rows, NT a lane: red[w][3][kAttemptRows].
template <int NT>
__device__ __forceinline__ void attempt_gravity(const PipeBufs& P, const GravTable& T, const double* tab, int st,
                                                int b0, int rows, int shares, int w, bool staged, double* red) {
    const int lane = threadIdx.x & 31;
    double px[NT], py[NT], pz[NT], a[NT][3];
    bool ok[NT];
#pragma unroll
    for (int q = 0; q < NT; ++q) {
        px[q] = 7000.0;  // a valid dummy position
        py[q] = 0.0;
        pz[q] = 0.0;
        ok[q] = attempt_position(P, st, b0, rows, q * 32 + lane, w == 0, staged, &px[q], &py[q], &pz[q]);
    }
    if (staged) gravity_part<NT>(tab, T.order, shares, 0, shares, w, px, py, pz, a);
#pragma unroll
    for (int q = 0; q < NT; ++q)
#pragma unroll
        for (int k = 0; k < 3; ++k) red[(w * 3 + k) * kAttemptRows + q * 32 + lane] = ok[q] ? a[q][k] : NAN;
}

// The same in the order of PropArgs::ordered: the columns in kGravityPartsMax
// runs (red[run][3][kAttemptRows]), warp w one run for one half of the rows.
__device__ __forceinline__ void attempt_gravity_cells(const PipeBufs& P, const GravTable& T, const double* tab, int st,
                                                      int b0, int rows, int w, bool staged, double* red) {
    const int run = w % kGravityPartsMax, r = w / kGravityPartsMax * 32 + (threadIdx.x & 31);
    if (w >= 2 * kGravityPartsMax || (r & ~31) >= rows) return;
    double x = 7000.0, y = 0.0, z = 0.0, a[1][3];
    const bool ok = attempt_position(P, st, b0, rows, r, run == 0, staged, &x, &y, &z);
    if (staged)
        gravity_columns<1>(tab, T.order, gravity_part_column(T.order, run, kGravityPartsMax),
                           gravity_part_column(T.order, run + 1, kGravityPartsMax), &x, &y, &z, a);
#pragma unroll
    for (int k = 0; k < 3; ++k) red[(run * 3 + k) * kAttemptRows + r] = ok ? a[0][k] : NAN;
}

}  // namespace

// Launch number `at` of six: up to `rounds` attempts of the rows of list at % 2,
// counted in count[at % 3]; rows that go on are appended to the other list and
// count[(at + 1) % 3], and count[(at + 2) % 3] is cleared for the launch after
// this one (nothing reads it any more).  Once the call's wall-clock limit is
// over no row makes another attempt: the rows go on to the next list as they
// are, until the host ends them (over[at % 2] is the launch before's word, read
// alike by every thread; over[(at + 1) % 2] is this one's).  `first`: one
// attempt whatever the clock says.
template <int M>
__global__ void __launch_bounds__(kAttemptThreads, 1)
    at_attempt(const __grid_constant__ PropArgs A, const __grid_constant__ PipeBufs P, int at, int dense,
               int rounds, int first) {
    extern __shared__ __align__(16) double smem_dyn[];  // [shares][3][kAttemptRows] sums, the table
    __shared__ __align__(8) uint64_t bar;
    __shared__ EclWarpStore ecl_ws[kAttemptRows / 32];
    // drag: rows above and below ~510 km; the counts of this stage and the next
    __shared__ int32_t n_list[2][2], row_list[2][kAttemptRows];
    // the CTA's trajectories, of this attempt and the next; row r is slot b0 + r
    __shared__ int32_t trajs[2][kAttemptRows], n_traj[2];
    __shared__ int32_t over;        // the call's wall-clock limit is over
    __shared__ int32_t four_lanes;  // exact density: the launch's rows a CTA are at most kFourLanesRows
    const int count = P.count[at % 3];
    const bool none = !first && P.over[at & 1];  // no attempt in this launch
    const int per = (count + gridDim.x - 1) / gridDim.x;
    const int b0 = blockIdx.x * per;
    int rows = min(per, count - b0);
    if (blockIdx.x == 0 && threadIdx.x == 0) P.count[(at + 2) % 3] = 0;
    if (rows <= 0) return;  // uniform across the CTA
    if (threadIdx.x < rows) trajs[0][threadIdx.x] = P.idx[at & 1][b0 + threadIdx.x];
    const ForceParams& fp = A.force;
    if (threadIdx.x == 0) four_lanes = per <= kFourLanesRows;
    const int tid = threadIdx.x, warp = tid >> 5;
    const int drag_warps = fp.drag ? kDragWarps : 0;
    const int shares = kAttemptThreads / 32 - drag_warps;
    double* red = smem_dyn;
    double* tab = smem_dyn + shares * 3 * kAttemptRows;
    bool staged = true;
    if (tid == 0) {
        over = none;
        if (none) P.over[(at & 1) ^ 1] = 1;
    }
    if (fp.gravity_on && !none)
        staged = stage_begin(&bar, A.grav.bytes, [&](auto copy) { copy(tab, A.grav.tab, A.grav.bytes); });
    const int stages = Tab<M>::S + (dense ? 1 : 0);
    __syncthreads();  // the trajectories are listed
    int round = 0;
    for (; round < rounds && rows > 0 && !over; ++round) {
        const int32_t* list = trajs[round & 1];
        if (tid == 0) n_traj[(round & 1) ^ 1] = 0;  // read again after the stages' barriers
        // the instants: part k of stage s of row r, the parts in different warps
        // (ordered rows: pl_times has run)
        if (!A.ordered) {
            const int items = rows * stages, padded = (items + 31) & ~31;
            for (int i = tid; i < 4 * padded; i += kAttemptThreads) {
                const int part = i / padded, k = i - part * padded;
                if (k >= items) continue;
                const int st = k / rows, slot = b0 + k - st * rows;
                const TrajState& s = P.st[list[slot - b0]];
                if (st == 0 && (s.flags & kHaveK1)) continue;
                times_row(A, P, s, slot, st, stage_time<M>(s, st), 1 << part);
            }
        }
        if (round == 0 && fp.gravity_on && staged) staged = stage_wait(&bar);
        for (int st = 0; st <= stages; ++st) {
            if (st == 0 && tid < 2) n_list[0][tid] = 0;
            __syncthreads();  // the last stage's sums and drag are there
            if (tid < 2) n_list[(st + 1) & 1][tid] = 0;
            if (tid < rows) {
                const int slot = b0 + tid;
                if (st > 0 && fp.gravity_on && !P.skip[slot]) {
                    const int sums = A.grav.cells ? kGravityPartsMax : shares;
                    for (int k = 0; k < 3; ++k) {
                        double g = red[k * kAttemptRows + tid];
                        for (int w = 1; w < sums; ++w) g += red[(w * 3 + k) * kAttemptRows + tid];
                        P.agrav[(size_t)k * P.cap + slot] = g;
                    }
                }
                double r2;
                if (st < stages && prep_row<M>(A, P, P.st[list[slot - b0]], slot, st, &r2) && fp.drag) {
                    const int c = sqrt(r2) - fp.earth_radius >= 510.0 ? 0 : 1;
                    row_list[c][atomicAdd(&n_list[st & 1][c], 1)] = tid;
                }
            }
            if (st == stages) break;
            __syncthreads();
            if (warp < drag_warps) {
                const int hi = n_list[st & 1][0], lo = n_list[st & 1][1];
                if (fp.atm_model == 4 && A.ordered) {
                    // as the stage kernels' lanes: one a row above, four below
                    attempt_drag<1, 3>(fp, P, st, b0, row_list[0], hi, row_list[1], 0);
                    attempt_drag<4, 3>(fp, P, st, b0, row_list[0], 0, row_list[1], lo);
                } else if (fp.atm_model == 4 && four_lanes)
                    attempt_drag<4, 0>(fp, P, st, b0, row_list[0], hi, row_list[1], lo);
                else if (fp.atm_model == 4)
                    attempt_drag<2, 0>(fp, P, st, b0, row_list[0], hi, row_list[1], lo);
                else if (fp.drag_fp32)
                    attempt_drag<1, 2>(fp, P, st, b0, row_list[0], hi, row_list[1], lo);
                else if (A.ordered)
                    attempt_drag<1, 1>(fp, P, st, b0, row_list[0], hi, row_list[1], lo);
                else
                    attempt_drag<4, 4>(fp, P, st, b0, row_list[0], hi, row_list[1], lo);
            } else if (fp.gravity_on) {
                if (A.grav.cells)
                    attempt_gravity_cells(P, A.grav, tab, st, b0, rows, warp - drag_warps, staged, red);
                else if (rows <= 32)
                    attempt_gravity<1>(P, A.grav, tab, st, b0, rows, shares, warp - drag_warps, staged, red);
                else
                    attempt_gravity<2>(P, A.grav, tab, st, b0, rows, shares, warp - drag_warps, staged, red);
            }
        }
        if (warp * 32 < rows)
            control_warp<M>(A, P, tid < rows ? list[tid] : 0, b0 + tid, tid < rows, trajs[(round & 1) ^ 1],
                            &n_traj[(round & 1) ^ 1], ecl_ws[warp], dense);
        // the clock, read by a warp that has no controller's rows
        if (tid == kAttemptThreads - 1 && over_time(A, P)) over = P.over[(at & 1) ^ 1] = 1;
        __syncthreads();
        rows = n_traj[(round & 1) ^ 1];
    }
    if (tid < rows) {
        const int i = atomicAdd(&P.count[(at + 1) % 3], 1);
        P.idx[(at & 1) ^ 1][i] = trajs[round & 1][tid];
    }
}

template <int M>
static cudaError_t run(const PropArgs& A, const PipeBufs& P, ReplayRes& R, cudaStream_t user, double max_seconds) {
    const bool dense = (A.out_mode != kOutFinalEci || A.force.srp) && !Tab<M>::FSAL;
    const int shares = kAttemptThreads / 32 - (A.force.drag ? kDragWarps : 0);
    const size_t smem = attempt_smem_bytes(A.grav, shares);
    cudaError_t e =
        cudaFuncSetAttribute(at_attempt<M>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kAttemptSmem);
    if (e == cudaSuccess) e = upload_fixed_fit(A, user);
    if (e != cudaSuccess) return e;
    const int blocks = (int)((A.n + kBlock - 1) / kBlock);
    const int ctas = (int)(A.n < device_sm_count() ? A.n : device_sm_count());
    // launches that make an attempt whatever the clock says: as many as the
    // stage kernels make before the host first looks at it
    int unconditional = 4;
    return replay(
        P, R, user, max_seconds, false, false, [&](cudaStream_t st) { pl_init<M><<<blocks, kBlock, 0, st>>>(A, P); },
        [&](cudaStream_t st, cudaStream_t, const StreamOrder&) {
            // six attempts bring the two lists and the three counters back
            for (int at = 0; at < 6; ++at) {
                if (A.ordered) launch_times(A, P, M, at & 1, at % 3, Tab<M>::S + (dense ? 1 : 0), st);
                at_attempt<M><<<ctas, kAttemptThreads, smem, st>>>(A, P, at, dense ? 1 : 0,
                                                                  A.ordered ? 1 : kAttemptRounds, unconditional > 0 ? 1 : 0);
                if (unconditional > 0) --unconditional;
            }
        },
        [&](cudaStream_t st) { pl_abort<M><<<blocks, kBlock, 0, st>>>(A, P, 0); }, [] {});
}

bool attempt_fits(const PropArgs& A) {
    if (A.sur.P || A.grav.ls > 0 || A.n > (int64_t)kAttemptRows * device_sm_count()) return false;
    return !A.force.gravity_on || attempt_smem_bytes(A.grav, kAttemptThreads / 32) <= kAttemptSmem;
}

cudaError_t launch_attempts(const PropArgs& A, const PipeBufs& P, ReplayRes& R, int method, cudaStream_t st,
                            double max_seconds) {
    switch (method) {
        case kDopri5: return run<kDopri5>(A, P, R, st, max_seconds);
        case kDop853: return run<kDop853>(A, P, R, st, max_seconds);
        case kDopri5Compat: return run<kDopri5Compat>(A, P, R, st, max_seconds);
        case kVern7: return run<kVern7>(A, P, R, st, max_seconds);
        case kVern9: return run<kVern9>(A, P, R, st, max_seconds);
        default: return cudaErrorInvalidValue;
    }
}

}  // namespace bqp
