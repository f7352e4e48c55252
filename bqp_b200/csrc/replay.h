// Host loop of the stage-synchronous engine: attempts issued until no row is
// active.
#pragma once
#include <cuda_runtime.h>

#include <chrono>
#include <cstdint>

#include "jb2008.cuh"
#include "launch.h"

namespace bqp {

// The fixed-node fits in this translation unit's constant memory: the same
// table for every context, ordered on the caller's stream before the call's
// kernels.
static inline cudaError_t upload_fixed_fit(const PropArgs& A, cudaStream_t user) {
    if (!A.force.fit) return cudaSuccess;
    if (!A.fit_host) return cudaErrorInvalidValue;
    return cudaMemcpyToSymbolAsync(jb::c_fixed_fit, A.fit_host, sizeof(jb::JbFit), 0, cudaMemcpyHostToDevice, user);
}

// Orders what follows on `after` behind what is on `before` (in a capture: an
// edge between the two streams' nodes).
struct StreamOrder {
    cudaEvent_t ev;
    void operator()(cudaStream_t before, cudaStream_t after) const {
        cudaEventRecord(ev, before);
        cudaStreamWaitEvent(after, ev, 0);
    }
};

// init(st) fills the first active list; enqueue(st, st2, order) issues some
// attempts, after which list 0 and count[0] are the active rows again --
// captured once as a graph and replayed (`graph`), or launched as they are (a
// few launches: cheaper than to instantiate a graph a call); abort(st) ends
// the rows of list 0.  timed: collect() reads each replay's events.
template <class Init, class Enqueue, class Abort, class Collect>
static cudaError_t replay(const PipeBufs& P, ReplayRes& R, cudaStream_t user, double max_seconds, bool graph_on,
                          bool timed, Init init, Enqueue enqueue, Abort abort, Collect collect) {
    // streams of the context's own, ordered after the caller's (graphs need a
    // capturable stream); the second one's kernels give way to the first's
    cudaError_t e = R.ready();
    if (e != cudaSuccess) return e;
    const cudaStream_t st = R.st, st2 = R.st2;
    const StreamOrder order{R.ev_order};
    cudaEventRecord(R.ev_in, user);
    cudaStreamWaitEvent(st, R.ev_in, 0);

    cudaMemsetAsync(P.count, 0, 3 * sizeof(int32_t), st);
    init(st);
    cudaGraph_t graph = nullptr;
    cudaGraphExec_t exec = nullptr;
    if (graph_on) {
        e = cudaStreamBeginCapture(st, cudaStreamCaptureModeThreadLocal);
        if (e == cudaSuccess) {
            enqueue(st, st2, order);
            e = cudaStreamEndCapture(st, &graph);
        }
        if (e == cudaSuccess) e = cudaGraphInstantiate(&exec, graph, 0);
    }
    auto issue = [&]() -> cudaError_t {
        if (graph_on) return cudaGraphLaunch(exec, st);
        enqueue(st, st2, order);
        return cudaGetLastError();
    };
    const auto t_start = std::chrono::steady_clock::now();
    // host loop: replay, keep one replay in flight ahead of the count check
    bool done = false;
    while (e == cudaSuccess && !done) {
        e = issue();
        if (e != cudaSuccess) break;
        cudaMemcpyAsync(R.h_count, &P.count[0], sizeof(int32_t), cudaMemcpyDeviceToHost, st);
        cudaEventRecord(R.ev_cnt, st);
        if (timed) {
            // no replay in flight while the events of this one are read
            e = cudaEventSynchronize(R.ev_cnt);
            if (e != cudaSuccess) break;
            collect();
        }
        e = issue();  // speculative: cheap when nothing is active
        if (e != cudaSuccess) break;
        e = cudaEventSynchronize(R.ev_cnt);
        if (timed && e == cudaSuccess) {
            e = cudaStreamSynchronize(st);
            if (e == cudaSuccess) collect();
        }
        if (*R.h_count == 0) done = true;
        const double elapsed =
            std::chrono::duration<double>(std::chrono::steady_clock::now() - t_start).count();
        if (!done && max_seconds > 0.0 && elapsed > max_seconds) {
            cudaStreamSynchronize(st);
            abort(st);
            done = true;
        }
    }
    if (e == cudaSuccess) e = cudaGetLastError();
    cudaEventRecord(R.ev_out, st);
    cudaStreamWaitEvent(user, R.ev_out, 0);
    cudaStreamSynchronize(st);
    if (exec) cudaGraphExecDestroy(exec);
    if (graph) cudaGraphDestroy(graph);
    return e;
}

}  // namespace bqp
