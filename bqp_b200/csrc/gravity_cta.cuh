// One CTA's (or cluster's) share of a gravity batch, used by the gravity-only
// kernel and by the stage-synchronous engine's gravity stage.
//
// FP64 field.  A warp carries 32 lanes x NT rows, which share its table reads
// from shared memory.  The warps of a CTA are cut into groups of `parts`; a
// group takes one tile of rows at a time, each warp its share of the columns
// (gravity_part), and one of them adds the shares in a fixed order.  A
// cluster of CTAs does the same with more shares: every CTA stages only its
// own columns, works on all rows of the cluster, and the CTAs' sums meet in
// one of them over distributed shared memory.  See gravity_launch and
// gravity_plan for how the split is picked.
//
// Split-precision field, and the FP64 field in the order of its cells
// (GravTable::cells): the CTA is cut into `parts` groups of `tpart`
// threads, every group evaluates all rows of a pass over its own run of
// columns, and the partial sums are added in shared memory.
#pragma once
#include <cuda_runtime.h>

#include "gravity.cuh"
#include "kernels.cuh"

namespace bqp {

// opt-in shared memory per CTA, less room for the static mbarrier
constexpr size_t kSmemPerBlock = 227 * 1024 - 64;
constexpr uint64_t kStageWaitNs = 1000000000ull;   // 1 s bound on the table copy
constexpr uint64_t kStageDrainNs = 2000000000ull;  // after a timeout: 2 s more for the copy to land

// Sticky flag of this translation unit's gravity kernels: set when a CTA's
// table copy did not land within kStageWaitNs.  Every later CTA (of this and
// later launches) then stages nothing and reports its rows lost, so no CTA
// starts on an SM where an earlier CTA's copy may still be writing shared
// memory.  It stays set until the process exits: a bulk copy that takes
// seconds means the device is not in a state to trust.
static __device__ unsigned int g_stage_fault = 0u;

// Copies from global into shared memory by the bulk-copy engine (addresses
// 16-byte aligned, sizes multiples of 16), completion signalled on an
// mbarrier.  stage_begin: every thread calls it once; `issue(copy)` runs in
// thread 0 and calls copy(dst, src, bytes) for every piece, `total` bytes in
// all.  False if an earlier CTA's copy was lost.  stage_wait: every thread
// waits for at most kStageWaitNs; all get false if any thread saw the copies
// unfinished then.  On that failure the CTA sets g_stage_fault and thread 0
// keeps the CTA resident for up to kStageDrainNs more, until the copies have
// landed, so the CTA does not exit with a copy in flight unless it never
// completes.
template <class Issue>
__device__ __forceinline__ bool stage_begin(uint64_t* bar, uint32_t total, Issue issue) {
    const uint32_t bar_a = (uint32_t)__cvta_generic_to_shared(bar);
    if (threadIdx.x == 0) {
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(bar_a) : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    // one read of the sticky flag decides for the whole CTA
    const bool faulted =
        __syncthreads_or(threadIdx.x == 0 && *static_cast<volatile unsigned int*>(&g_stage_fault) != 0u);
    if (faulted) return false;
    if (threadIdx.x == 0) {
        asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar_a), "r"(total) : "memory");
        issue([&](void* smem_dst, const void* gsrc, uint32_t bytes) {
            const uint32_t dst_a = (uint32_t)__cvta_generic_to_shared(smem_dst);
            constexpr uint32_t kChunk = 32768;
            for (uint32_t off = 0; off < bytes; off += kChunk) {
                const uint32_t n = bytes - off < kChunk ? bytes - off : kChunk;
                asm volatile(
                    "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                        dst_a + off),
                    "l"(static_cast<const char*>(gsrc) + off), "r"(n), "r"(bar_a)
                    : "memory");
            }
        });
    }
    return true;
}

__device__ __forceinline__ bool stage_landed(uint32_t bar_a, uint64_t limit_ns) {
    uint32_t done = 0;
    uint64_t t0 = 0;
    for (uint32_t it = 0;; ++it) {
        asm volatile(
            "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], 0;\n\tselp.u32 %0, 1, 0, "
            "p;\n\t}"
            : "=r"(done)
            : "r"(bar_a)
            : "memory");
        if (done) return true;
        if ((it & 255u) == 255u) {
            const uint64_t t = global_ns();
            if (t0 == 0) t0 = t;
            else if (t - t0 > limit_ns) return false;
        }
    }
}

__device__ __forceinline__ bool stage_wait(uint64_t* bar) {
    const uint32_t bar_a = (uint32_t)__cvta_generic_to_shared(bar);
    // one verdict for the whole CTA (a thread may give up just before the
    // copies land while another sees them land)
    if (!__syncthreads_or(!stage_landed(bar_a, kStageWaitNs))) return true;
    if (threadIdx.x == 0) {
        atomicExch(&g_stage_fault, 1u);
        stage_landed(bar_a, kStageDrainNs);
    }
    __syncthreads();
    return false;
}
constexpr int kGravityPartsMax = 4;

struct GravLayout {
    int tpart;  // threads per group (a multiple of 32, at most the CTA)
    int parts;  // groups
};

BQP_HD GravLayout gravity_layout(int rows, int nt, int block, int parts_max) {
    const int need = (rows + nt - 1) / nt;
    int tpart = (need + 31) / 32 * 32;
    if (tpart > block) tpart = block;
    if (tpart < 32) tpart = 32;
    int parts = block / tpart;
    if (parts > parts_max) parts = parts_max;
    if (parts < 1) parts = 1;
    return {tpart, parts};
}

// The field table as the gravity kernels see it.  Plain form (ls = 0): the
// FP64 table of gravity_part.  Split form (ls > 0): the FP64 cells of rows
// <= ls followed by the FP32 cells of the rest (gravity_columns_split).
struct GravTable {
    const double* tab;
    int order;
    int ls;          // 0: plain FP64; else the last FP64 row
    uint32_t bytes;  // size of tab (plain form: without its pad)
    int in_smem;     // split form and cells: 1 if staged into shared memory per CTA
    int cells;       // 1: plain FP64 cells {a, b, Ax .. Bz} (gravity_columns), in every column
};

inline uint32_t gravity_table_bytes(int order, int ls) {
    return (uint32_t)(split_lo_cells(ls) * kCellDoubles * sizeof(double) +
                      split_hi_cells(order, ls) * kCellDoubles * sizeof(float));
}

// The plain form's view of an FP64 table.
inline GravTable gravity_table(const double* tab, int order) {
    GravTable T{};
    T.tab = tab;
    T.order = order;
    T.bytes = (uint32_t)(gravity_tab_doubles(order) * sizeof(double));
    T.in_smem = 1;
    return T;
}

// The run of columns (first, how many; 0: none) that shares wa .. wa + own - 1
// own in block k; false past the last block.
BQP_HD bool gravity_run(int order, int shares, int wa, int own, int k, int* j, int* n) {
    const int ncol = order + 2;
    *j = gravity_share_column(shares, k, (k & 1) ? wa + own - 1 : wa);
    *n = *j >= ncol ? 0 : (*j + own < ncol ? own : ncol - *j);
    return k * shares < ncol;
}
BQP_HD int gravity_run_doubles(int order, int j, int n) {
    return gravity_tab_offset(order, j + n) - gravity_tab_offset(order, j);
}

// Shared memory of a CTA's columns of an FP64 table, the largest over the
// cluster's CTAs, without the pad.
inline size_t gravity_run_bytes(int order, int cluster, int warps) {
    if (cluster == 1) return gravity_tab_doubles(order) * sizeof(double);
    size_t most = 0;
    for (int r = 0; r < cluster; ++r) {
        size_t b = 0;
        int j, m;
        for (int k = 0; gravity_run(order, cluster * warps, r * warps, warps, k, &j, &m); ++k)
            if (m > 0) b += (size_t)gravity_run_doubles(order, j, m) * sizeof(double);
        most = b > most ? b : most;
    }
    return most;
}

// Partial sums of a CTA's tiles (twice: the next tile's are written while one
// warp still adds) and, in a cluster, of its CTAs' (twice again).
BQP_HD int gravity_red_doubles(int cluster, int warps, int nt) {
    return 2 * warps * nt * 96 + (cluster > 1 ? 2 * cluster * nt * 96 : 0);
}

constexpr int kGravityClusterMax = 8;

// Warps that share a tile's columns, for a CTA of `warps` warps with `rows`
// rows: the power of two (or all warps) whose rounds cost least, in cells of
// one row a lane.  A round costs its share of the cells (never less than the
// longest column) plus the set-up of a share -- the position, its powers, the
// columns' ends: about 20 cells -- and, where warps share a tile, the sums
// over the shares and the barrier (about 2 cells a share).  The same for all
// CTAs of a launch, so that a row's result does not depend on which one it is
// in.
BQP_HD int gravity_plan(int order, int rows, int warps, int nt) {
    const unsigned cells = gravity_cells(order), tile = 32 * nt, longest = order + 2;
    unsigned best = warps, least = 0xffffffffu;
    for (unsigned parts = 1;; parts *= 2) {
        if (parts > (unsigned)warps) break;
        if (warps % parts) parts = warps;  // the last one
        unsigned share = (cells + parts - 1) / parts;
        share = (share > longest ? share : longest) + 20 + (parts > 1 ? 2 * parts : 0);
        const unsigned pass = tile * (warps / parts);
        const unsigned full = rows / pass, rest = rows - full * pass;
        const unsigned cost = (full * nt + (rest > tile ? (unsigned)nt : (rest + 31) / 32)) * share;
        if (cost < least) {
            least = cost;
            best = parts;
        }
    }
    return (int)best;
}

__device__ __forceinline__ uint32_t cluster_rank() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ void cluster_arrive() {
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
}
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }
// To the same place in the shared memory of the cluster's CTA `rank`.
__device__ __forceinline__ uint32_t cluster_address(const void* local, uint32_t rank) {
    uint32_t a;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;"
                 : "=r"(a)
                 : "r"((uint32_t)__cvta_generic_to_shared(local)), "r"(rank));
    return a;
}
__device__ __forceinline__ void cluster_store(double* local, uint32_t rank, double v) {
    asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(cluster_address(local, rank)), "d"(v) : "memory");
}
__device__ __forceinline__ void cluster_store(int* local, uint32_t rank, int v) {
    asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(cluster_address(local, rank)), "r"(v) : "memory");
}

// What one warp does for one tile: NT rows a lane from row `base` on (rows
// past b1 idle), share w of its group.  `red` is the group's area of this
// round, [share][q][3][lane].  Warp `adder` of the group adds the shares in
// the order of w; tail(on, sums, whether this warp holds them) follows in
// every warp.  Every thread of the CTA reaches the one barrier (none with one
// share).
struct GravShare {
    const double* tab;  // the CTA's columns
    int order, shares, wa, own;  // all shares, and the CTA's
    int parts, w;                // the group's shares, this warp's
    bool staged;                 // false: the table copy was lost
};
template <int NT, class Load, class Tail>
__device__ __forceinline__ void gravity_tile(const GravShare& G, int base, int b1, double* red, int adder, Load& load,
                                             Tail tail) {
    const int lane = threadIdx.x & 31;
    double px[NT], py[NT], pz[NT], a[NT][3];
    bool on[NT];
#pragma unroll
    for (int q = 0; q < NT; ++q) {
        const int i = base + q * 32 + lane;
        px[q] = 7000.0;  // a valid dummy position for idle lanes
        py[q] = 0.0;
        pz[q] = 0.0;
        on[q] = i < b1 && load(i, px[q], py[q], pz[q]);
    }
    if (G.staged) {
        gravity_part<NT>(G.tab, G.order, G.shares, G.wa, G.own, G.wa + G.w, px, py, pz, a);
    } else {
#pragma unroll
        for (int q = 0; q < NT; ++q) a[q][0] = a[q][1] = a[q][2] = NAN;
    }
    const bool mine = G.w == adder;
    if (G.parts > 1) {
        if (!mine) {
#pragma unroll
            for (int q = 0; q < NT; ++q)
#pragma unroll
                for (int k = 0; k < 3; ++k) red[((G.w * NT + q) * 3 + k) * 32 + lane] = a[q][k];
        }
        __syncthreads();
        if (mine) {
            double own[NT][3];
#pragma unroll
            for (int q = 0; q < NT; ++q)
#pragma unroll
                for (int k = 0; k < 3; ++k) {
                    own[q][k] = a[q][k];
                    a[q][k] = 0.0;
                }
            for (int p = 0; p < G.parts; ++p) {
#pragma unroll
                for (int q = 0; q < NT; ++q)
#pragma unroll
                    for (int k = 0; k < 3; ++k)
                        a[q][k] += p == G.w ? own[q][k] : red[((p * NT + q) * 3 + k) * 32 + lane];
            }
        }
    }
    tail(on, a, mine);
}

// Rows [b0, b1) of this CTA or cluster; the plan (and so the order in which a
// row's column sums are added) follows layout_rows, the same for every CTA of
// a launch.  load(i, x, y, z) fetches row i's Earth-fixed position and returns
// false for a row to leave out (it records that row's outcome itself; every
// share calls it, so it must be idempotent).  store(i, a) receives the field
// of row i.  lost(i) records that row i got no field because a table copy did
// not complete in time.
template <int NT, bool kCluster, class Load, class Store, class Lost>
__device__ __forceinline__ void gravity_cta_plain(const GravTable& T, int cluster, int layout_rows, int b0, int b1,
                                                  Load load, Store store, Lost lost) {
    extern __shared__ __align__(16) double smem_dyn[];
    __shared__ __align__(8) uint64_t bar;
    __shared__ int landed[kGravityClusterMax];  // each CTA's verdict on its copy
    const int warps = blockDim.x >> 5, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int ncta = kCluster ? cluster : 1;
    const int rank = kCluster ? (int)cluster_rank() : 0;
    // [2][warps][NT][3][32] shares' sums, [2][ncta][NT][3][32] CTAs' sums, the columns
    double* red = smem_dyn;
    const int half = warps * NT * 96;
    double* cross = red + 2 * half;
    const int chalf = ncta * NT * 96;
    double* tab = smem_dyn + gravity_red_doubles(ncta, warps, NT);
    const int all = ncta * warps;  // the shares of a cluster
    uint32_t total = T.bytes;
    if (kCluster) {
        total = 0;
        int j, m;
        for (int k = 0; gravity_run(T.order, all, rank * warps, warps, k, &j, &m); ++k)
            if (m > 0) total += (uint32_t)gravity_run_doubles(T.order, j, m) * 8u;
    }
    GravShare G;
    G.tab = tab;
    G.order = T.order;
    G.staged = stage_begin(&bar, total, [&](auto copy) {
        if (!kCluster) {
            copy(tab, T.tab, total);
            return;
        }
        double* dst = tab;
        int j, m;
        for (int k = 0; gravity_run(T.order, all, rank * warps, warps, k, &j, &m); ++k) {
            if (m <= 0) continue;
            const int len = gravity_run_doubles(T.order, j, m);
            copy(dst, T.tab + gravity_tab_offset(T.order, j), (uint32_t)len * 8u);
            dst += len;
        }
    });
    if (kCluster) cluster_arrive();  // this CTA's shared memory may be written to
    G.parts = kCluster ? warps : gravity_plan(T.order, layout_rows, warps, NT);
    const int groups = warps / G.parts, group = warp / G.parts;
    G.w = warp - group * G.parts;
    G.shares = kCluster ? all : G.parts;
    G.wa = kCluster ? rank * warps : 0;
    G.own = G.parts;
    if (G.staged) G.staged = stage_wait(&bar);  // the verdict is the same in every thread
    if (kCluster) {
        cluster_wait();
        if (threadIdx.x < (unsigned)ncta) cluster_store(&landed[rank], threadIdx.x, G.staged ? 1 : 0);
        cluster_arrive();
    } else if (!G.staged) {
        for (int i = b0 + threadIdx.x; i < b1; i += blockDim.x) lost(i);
        return;
    }
    const int tile = 32 * NT;
    int round = 0, base = 0;
    // the CTAs' sums of round r (its rows from `from` on), added by CTA
    // r % ncta in the order of ranks
    auto finish = [&](int r, int from) {
        if (warp != 0 || r % ncta != rank) return;
        bool ok = true;
        for (int c = 0; c < ncta; ++c) ok = ok && landed[c] != 0;
        const double* x = cross + (r & 1) * chalf + lane;
#pragma unroll
        for (int q = 0; q < NT; ++q) {
            const int i = from + q * 32 + lane;
            if (i >= b1) continue;
            double px, py, pz, a[3] = {0.0, 0.0, 0.0};
            for (int c = 0; c < ncta; ++c)
                for (int k = 0; k < 3; ++k) a[k] += x[((c * NT + q) * 3 + k) * 32];
            if (!load(i, px, py, pz)) continue;
            if (ok) store(i, a);
            else lost(i);
        }
    };
    auto tail = [&](const auto& on, const auto& a, bool mine) {
        constexpr int nq = sizeof(on) / sizeof(bool);
        if (!kCluster) {
            if (mine) {
#pragma unroll
                for (int q = 0; q < nq; ++q)
                    if (on[q]) store(base + q * 32 + lane, a[q]);
            }
            return;
        }
        // round by round: wait for the sums of the round before (and so for
        // their area to be free two rounds on), add them, hand over this one's
        cluster_wait();
        if (round > 0) finish(round - 1, base - tile);
        if (mine) {
            double* x = cross + (round & 1) * chalf + rank * NT * 96 + lane;
#pragma unroll
            for (int q = 0; q < nq; ++q)
#pragma unroll
                for (int k = 0; k < 3; ++k) cluster_store(x + (q * 3 + k) * 32, round % ncta, a[q][k]);
        }
        cluster_arrive();
    };
    for (int base0 = b0; base0 < b1; base0 += tile * groups, ++round) {
        base = base0 + group * tile;
        const int nt = base < b1 ? min(NT, (b1 - base + 31) >> 5) : 0;
        double* area = red + (round & 1) * half + group * G.parts * NT * 96;
        const int adder = round % G.parts;
        // fewer rows a lane in a tile that is not full
        if (nt == NT) gravity_tile<NT>(G, base, b1, area, adder, load, tail);
        else if (NT > 3 && nt == 3) gravity_tile<3>(G, base, b1, area, adder, load, tail);
        else if (NT > 2 && nt == 2) gravity_tile<2>(G, base, b1, area, adder, load, tail);
        else if (NT > 1 && nt == 1) gravity_tile<1>(G, base, b1, area, adder, load, tail);
        else if (G.parts > 1) __syncthreads();  // a group without rows keeps the barrier count
    }
    if (kCluster) {
        cluster_wait();
        finish(round - 1, base);
    }
}

template <int NT, class Load, class Store, class Lost>
__device__ __forceinline__ void gravity_cta_split(const GravTable& T, int parts_max, int layout_rows, int b0, int b1,
                                                  Load load, Store store, Lost lost) {
    extern __shared__ __align__(16) double smem_dyn[];
    __shared__ __align__(8) uint64_t bar;
    const GravLayout L = gravity_layout(layout_rows, NT, blockDim.x, parts_max);
    if (T.in_smem && !(stage_begin(&bar, T.bytes, [&](auto copy) { copy(smem_dyn, T.tab, T.bytes); }) &&
                       stage_wait(&bar))) {
        for (int i = b0 + threadIdx.x; i < b1; i += blockDim.x) lost(i);
        return;  // the verdict is the same in every thread
    }
    const int order = T.order;
    const double* __restrict__ gtab = T.tab;
    double* red = smem_dyn + (T.in_smem ? T.bytes / sizeof(double) : 0);
    const int part = threadIdx.x / L.tpart;
    const int tid = threadIdx.x - part * L.tpart;
    const bool member = part < L.parts;
    const int j0 = gravity_part_column(order, part, L.parts);
    const int j1 = gravity_part_column(order, part + 1, L.parts);
    const int per_pass = L.tpart * NT;
    for (int base = b0; base < b1; base += per_pass) {
        double px[NT], py[NT], pz[NT], a[NT][3];
        bool on[NT];
#pragma unroll
        for (int q = 0; q < NT; ++q) {
            const int i = base + q * L.tpart + tid;
            px[q] = 7000.0;  // a valid dummy position for idle lanes
            py[q] = 0.0;
            pz[q] = 0.0;
            on[q] = member && i < b1 && load(i, px[q], py[q], pz[q]);
        }
        if (member) {
            const size_t lo_doubles = (size_t)split_lo_cells(T.ls) * kCellDoubles;
            if (T.cells && T.in_smem)
                gravity_columns<NT>(smem_dyn, order, j0, j1, px, py, pz, a);
            else if (T.cells)
                gravity_columns<NT>(gtab, order, j0, j1, px, py, pz, a);
            else if (T.in_smem)
                gravity_columns_split<NT>(smem_dyn, reinterpret_cast<const float*>(smem_dyn + lo_doubles), order, T.ls,
                                          j0, j1, px, py, pz, a);
            else
                gravity_columns_split<NT>(gtab, reinterpret_cast<const float*>(gtab + lo_doubles), order, T.ls, j0, j1,
                                          px, py, pz, a);
        }
        if (L.parts > 1) {
            if (member && part > 0) {
#pragma unroll
                for (int q = 0; q < NT; ++q)
                    for (int c = 0; c < 3; ++c)
                        red[((size_t)(part - 1) * per_pass + q * L.tpart + tid) * 3 + c] = a[q][c];
            }
            __syncthreads();
            if (part == 0) {
                for (int g = 1; g < L.parts; ++g) {
#pragma unroll
                    for (int q = 0; q < NT; ++q)
                        for (int c = 0; c < 3; ++c)
                            a[q][c] += red[((size_t)(g - 1) * per_pass + q * L.tpart + tid) * 3 + c];
                }
            }
            __syncthreads();  // the area is reused by the next pass
        }
        if (part == 0) {
#pragma unroll
            for (int q = 0; q < NT; ++q)
                if (on[q]) store(base + q * L.tpart + tid, a[q]);
        }
    }
}

// The forms of the gravity kernels.
enum GravForm : int { kGravPlain = 0, kGravCluster = 1, kGravSplit = 2 };

// The rows of this CTA (its cluster) of n: equal shares of the launch.
template <int kForm>
__device__ __forceinline__ void gravity_rows(int64_t n, int cluster, int64_t* per, int64_t* c0, int64_t* c1) {
    const int64_t units = kForm == kGravCluster ? gridDim.x / cluster : gridDim.x;
    const int64_t unit = kForm == kGravCluster ? blockIdx.x / cluster : blockIdx.x;
    *per = (n + units - 1) / units;
    *c0 = unit * *per;
    *c1 = *c0 + *per < n ? *c0 + *per : n;
}

// aux: CTAs of a cluster (kGravCluster) or the most column groups (kGravSplit).
template <int NT, int kForm, class Load, class Store, class Lost>
__device__ __forceinline__ void gravity_cta(const GravTable& T, int aux, int layout_rows, int b0, int b1, Load load,
                                            Store store, Lost lost) {
    if (kForm == kGravSplit) gravity_cta_split<NT>(T, aux, layout_rows, b0, b1, load, store, lost);
    else gravity_cta_plain<NT, kForm == kGravCluster>(T, aux, layout_rows, b0, b1, load, store, lost);
}

// How a gravity kernel is launched: its form, CTAs of a cluster (1: none),
// rows a lane, threads, the most units (CTAs or clusters) at once, dynamic
// shared memory; `aux` of gravity_cta.
struct GravLaunch {
    int form, cluster, nt, threads, units, aux;
    size_t smem;
    // units for n rows: each with at least 8, since it stages the table
    // whatever its rows
    int grid(int64_t n) const {
        const int64_t want = (n + 7) / 8;
        return (int)(want < units ? (want < 1 ? 1 : want) : units) * cluster;
    }
};

// For up to n rows, with threads a CTA and rows a lane as configured (0: 256
// and 4).
//
// Clusters: where rows are few, a CTA's time is its columns' (whatever their
// rows, up to 32) and the staging of its table, and a cluster of four cuts
// both.  70x70, 1,000 rows: 14.0 us against 21.8 without; 2,000: 15.1 and
// 21.7; 3,000: 19.4 and 22.1; 4,000: 21.9 and 21.4, and beyond that rows are
// spread more evenly over 148 CTAs than over the 33 clusters of four that the
// chip holds (65,536 rows: 130 us in single CTAs, 188 in clusters of four).
// 40x40, 1,000 rows: 11.7 and 13.8; 2,000: 14.0 and 13.8; at 20x20 a table of
// 13 KB, clusters gain nothing.  Orders whose table does not fit beside the
// sums (79 and up) take the fewest CTAs that hold it: 120x120, 100,000 rows:
// 587 us in clusters of three, 602 of four (1,044 us when the table was read
// from L2).
inline GravLaunch gravity_launch(const GravTable& T, int64_t n, int sms, int threads, int slots) {
    GravLaunch G{};
    G.cluster = 1;
    G.nt = slots == 1 || slots == 2 ? slots : 4;
    if (threads <= 0 || threads > 256) threads = 256;
    if (threads < 32) threads = 32;
    G.threads = threads / 32 * 32;
    const int warps = G.threads / 32;
    if (T.ls > 0 || T.cells) {
        G.form = kGravSplit;
        G.units = sms;
        for (G.aux = kGravityPartsMax;; G.aux = 1) {
            G.smem = (T.in_smem ? T.bytes : 0) +
                     (G.aux > 1 ? (size_t)(G.threads - 32) * G.nt * 3 * sizeof(double) : 0);
            if (G.smem <= kSmemPerBlock || G.aux == 1) break;
        }
        return G;
    }
    if (T.order >= 40 && n <= (T.order >= 60 ? 3000 : 1500)) G.cluster = 4;
    for (;; ++G.cluster) {
        G.smem = gravity_run_bytes(T.order, G.cluster, warps) +
                 ((size_t)gravity_red_doubles(G.cluster, warps, G.nt) + kGravityTabPad) * sizeof(double);
        if (G.smem <= kSmemPerBlock || G.cluster == kGravityClusterMax) break;
    }
    G.form = G.cluster > 1 ? kGravCluster : kGravPlain;
    G.aux = G.cluster;
    G.units = sms / G.cluster;
    return G;
}

// Launches a gravity kernel of G's form over `ctas` CTAs (whole clusters).
template <class... Params, class... Args>
cudaError_t gravity_run(const GravLaunch& G, void (*ker)(Params...), int ctas, cudaStream_t st, Args... args) {
    cudaLaunchAttribute at{};
    at.id = cudaLaunchAttributeClusterDimension;
    at.val.clusterDim.x = (unsigned)G.cluster;
    at.val.clusterDim.y = at.val.clusterDim.z = 1;
    cudaLaunchConfig_t c{};
    c.gridDim = dim3((unsigned)ctas);
    c.blockDim = dim3((unsigned)G.threads);
    c.dynamicSmemBytes = G.smem;
    c.stream = st;
    c.attrs = &at;
    c.numAttrs = G.cluster > 1 ? 1 : 0;
    return cudaLaunchKernelEx(&c, ker, Params(args)...);
}

// Readies a kernel for G: its shared memory (the bound, see kSmemLimit) and,
// for clusters, how many the device holds at once (fewer than SMs / CTAs where
// a GPC's SMs do not divide).
template <class... Params>
cudaError_t gravity_ready(GravLaunch& G, void (*ker)(Params...)) {
    if (G.smem > kSmemPerBlock) return cudaErrorInvalidValue;
    cudaError_t e = cudaFuncSetAttribute(ker, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmemPerBlock);
    if (e != cudaSuccess || G.cluster == 1) return e;
    cudaLaunchAttribute at{};
    at.id = cudaLaunchAttributeClusterDimension;
    at.val.clusterDim.x = (unsigned)G.cluster;
    at.val.clusterDim.y = at.val.clusterDim.z = 1;
    cudaLaunchConfig_t c{};
    c.gridDim = dim3((unsigned)(G.units * G.cluster));
    c.blockDim = dim3((unsigned)G.threads);
    c.dynamicSmemBytes = G.smem;
    c.attrs = &at;
    c.numAttrs = 1;
    int fit = 0;
    e = cudaOccupancyMaxActiveClusters(&fit, ker, &c);
    if (e == cudaSuccess && fit > 0 && fit < G.units) G.units = fit;
    return e;
}

}  // namespace bqp
