// Host test of lbm_b200/csrc/capture.hpp with a fake of the runtime calls it
// makes: whichever of them fails, the error reaches the caller, the capture
// has ended and no graph is left.  Exit code 0 on success.
#include <cstdio>

#include "../../lbm_b200/csrc/capture.hpp"

namespace {

cudaError_t begin_result, pending, end_result;
bool capturing = false, end_gives_graph = true;
int graphs = 0, ended = 0;

void reset()
{
    begin_result = pending = end_result = cudaSuccess;
    capturing = false;
    end_gives_graph = true;
    graphs = ended = 0;
}

}  // namespace

extern "C" {
cudaError_t cudaStreamBeginCapture(cudaStream_t, cudaStreamCaptureMode)
{
    capturing = begin_result == cudaSuccess;
    return begin_result;
}
cudaError_t cudaGetLastError()
{
    const cudaError_t e = pending;
    pending = cudaSuccess;
    return e;
}
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t* graph)
{
    ++ended;
    capturing = false;
    if (end_gives_graph) {
        *graph = reinterpret_cast<cudaGraph_t>(&graphs);
        ++graphs;
    }
    return end_result;
}
cudaError_t cudaGraphDestroy(cudaGraph_t)
{
    --graphs;
    return cudaSuccess;
}
}

int main()
{
    cudaGraph_t graph = nullptr;
    const auto fine = [] { return cudaSuccess; };
    // all well: the graph is the caller's
    reset();
    if (lbm::capture_graph(nullptr, &graph, fine) != cudaSuccess || !graph || graphs != 1 || ended != 1) return 1;
    // the capture does not start: nothing is launched
    reset();
    begin_result = cudaErrorIllegalState;
    bool ran = false;
    const auto mark = [&] {
        ran = true;
        return cudaSuccess;
    };
    if (lbm::capture_graph(nullptr, &graph, mark) != cudaErrorIllegalState || graph || ran || ended) return 2;
    // a refused launch: the capture itself ends well
    reset();
    const auto refused = [] {
        pending = cudaErrorInvalidConfiguration;
        return cudaSuccess;
    };
    if (lbm::capture_graph(nullptr, &graph, refused) != cudaErrorInvalidConfiguration || graph || graphs || ended != 1 ||
        pending != cudaSuccess)
        return 3;
    // a launch refused ahead of the capture, not looked at yet: reported as well
    reset();
    pending = cudaErrorInvalidValue;
    if (lbm::capture_graph(nullptr, &graph, fine) != cudaErrorInvalidValue || graph || graphs || ended != 1) return 6;
    // a failing copy among the launches
    reset();
    const auto copy = [] { return cudaErrorInvalidValue; };
    if (lbm::capture_graph(nullptr, &graph, copy) != cudaErrorInvalidValue || graph || graphs || ended != 1) return 4;
    // the capture was invalidated
    reset();
    end_result = cudaErrorStreamCaptureInvalidated;
    end_gives_graph = false;
    if (lbm::capture_graph(nullptr, &graph, fine) != cudaErrorStreamCaptureInvalidated || graph || capturing) return 5;
    std::puts("capture ok");
    return 0;
}
