// Host loop of the stage-synchronous engine: a graph of attempts, captured
// once a call and replayed until no row is active.
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

// init(st) fills the first active list; enqueue(st, st2, order) captures the
// graph, after which list 0 and count[0] are the active rows again; abort(st)
// ends the rows of list 0.  timed: collect() reads each replay's events.
template <class Init, class Enqueue, class Abort, class Collect>
static cudaError_t replay(const PropArgs& A, const PipeBufs& P, cudaStream_t user, double max_seconds, bool timed,
                          Init init, Enqueue enqueue, Abort abort, Collect collect) {
    (void)A;
    // private stream ordered after the caller's stream (graphs need a
    // capturable stream), and a second one, whose kernels give way to the
    // first's
    int prio_low = 0, prio_high = 0;
    cudaDeviceGetStreamPriorityRange(&prio_low, &prio_high);
    cudaStream_t st, st2;
    cudaError_t e = cudaStreamCreateWithPriority(&st, cudaStreamNonBlocking, prio_high);
    if (e != cudaSuccess) return e;
    e = cudaStreamCreateWithPriority(&st2, cudaStreamNonBlocking, prio_low);
    if (e != cudaSuccess) {
        cudaStreamDestroy(st);
        return e;
    }
    cudaEvent_t ev_in, ev_out, ev_cnt, ev_order;
    cudaEventCreateWithFlags(&ev_in, cudaEventDisableTiming);
    cudaEventCreateWithFlags(&ev_out, cudaEventDisableTiming);
    cudaEventCreateWithFlags(&ev_cnt, cudaEventDisableTiming);
    cudaEventCreateWithFlags(&ev_order, cudaEventDisableTiming);
    cudaEventRecord(ev_in, user);
    cudaStreamWaitEvent(st, ev_in, 0);
    int32_t* h_count = nullptr;
    cudaMallocHost(&h_count, sizeof(int32_t));

    cudaMemsetAsync(P.count, 0, 3 * sizeof(int32_t), st);
    init(st);
    cudaGraph_t graph = nullptr;
    cudaGraphExec_t exec = nullptr;
    e = cudaStreamBeginCapture(st, cudaStreamCaptureModeThreadLocal);
    if (e == cudaSuccess) {
        enqueue(st, st2, StreamOrder{ev_order});
        e = cudaStreamEndCapture(st, &graph);
    }
    if (e == cudaSuccess) e = cudaGraphInstantiate(&exec, graph, 0);
    const auto t_start = std::chrono::steady_clock::now();
    // host loop: replay, keep one replay in flight ahead of the count check
    bool done = false;
    while (e == cudaSuccess && !done) {
        e = cudaGraphLaunch(exec, st);
        if (e != cudaSuccess) break;
        cudaMemcpyAsync(h_count, &P.count[0], sizeof(int32_t), cudaMemcpyDeviceToHost, st);
        cudaEventRecord(ev_cnt, st);
        if (timed) {
            // no replay in flight while the events of this one are read
            e = cudaEventSynchronize(ev_cnt);
            if (e != cudaSuccess) break;
            collect();
        }
        e = cudaGraphLaunch(exec, st);  // speculative: cheap when nothing is active
        if (e != cudaSuccess) break;
        e = cudaEventSynchronize(ev_cnt);
        if (timed && e == cudaSuccess) {
            e = cudaStreamSynchronize(st);
            if (e == cudaSuccess) collect();
        }
        if (*h_count == 0) done = true;
        const double elapsed =
            std::chrono::duration<double>(std::chrono::steady_clock::now() - t_start).count();
        if (!done && max_seconds > 0.0 && elapsed > max_seconds) {
            cudaStreamSynchronize(st);
            abort(st);
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
    cudaEventDestroy(ev_in);
    cudaEventDestroy(ev_out);
    cudaEventDestroy(ev_cnt);
    cudaEventDestroy(ev_order);
    cudaStreamDestroy(st2);
    cudaStreamDestroy(st);
    return e;
}

}  // namespace bqp
