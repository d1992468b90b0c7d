// capture.hpp -- stream capture of a run of launches, every error of which
// reaches the caller.
//
// A launch that the runtime refuses while a stream captures leaves no node in
// the graph and does not end the capture: the only trace is cudaGetLastError().
// A graph taken without looking there would run without that kernel.
//
// Header-only, on the runtime's host interface alone, so the host tests can
// drive it with failing calls (tests/cpp/capture_test.cpp).
#pragma once

#include <cuda_runtime_api.h>

namespace lbm {

// Captures what enqueue() -> cudaError_t launches on st; *graph is the caller's
// to destroy on cudaSuccess, null otherwise.  Returns the first error of the
// capture's start, enqueue, its launches (or one not looked at before them) and
// the capture's end; st does not capture afterwards.
template <class F>
cudaError_t capture_graph(cudaStream_t st, cudaGraph_t* graph, F&& enqueue)
{
    *graph = nullptr;
    cudaError_t e = cudaStreamBeginCapture(st, cudaStreamCaptureModeThreadLocal);
    if (e != cudaSuccess) return e;
    e = enqueue();
    const cudaError_t launch = cudaGetLastError();
    const cudaError_t end = cudaStreamEndCapture(st, graph);
    if (e == cudaSuccess) e = launch;
    if (e == cudaSuccess) e = end;
    if (e != cudaSuccess) {
        if (*graph) cudaGraphDestroy(*graph);
        *graph = nullptr;
        cudaGetLastError();
    }
    return e;
}

}  // namespace lbm
