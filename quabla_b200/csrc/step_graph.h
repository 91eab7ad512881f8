// A kernel sequence launched as one CUDA graph, or launch by launch where it cannot be captured.
#pragma once
#include <cuda_runtime.h>

#include <cstdint>

namespace qb {

struct StepGraph {
    int uses = 0;
    cudaGraphExec_t exec = nullptr;
    int64_t launches = 0;
    bool single = false;  // capturing it failed once (no memory for the graph, say): launch by launch from then on
};

// Captures what `enqueue` (true: all of it queued) puts on `stream` into graph.exec.  False when any part of that fails:
// nothing has run, no capture is left open, no error is left pending, and the caller launches one by one.
template <typename Enqueue>
bool capture_sequence(cudaStream_t stream, StepGraph& graph, Enqueue&& enqueue) {
    graph.single = true;
    if (cudaStreamBeginCapture(stream, cudaStreamCaptureModeThreadLocal) != cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    const bool queued = enqueue();
    cudaGraph_t captured = nullptr;
    const cudaError_t ended = cudaStreamEndCapture(stream, &captured);
    if (queued && ended == cudaSuccess && cudaGraphInstantiate(&graph.exec, captured, 0) == cudaSuccess)
        graph.single = false;
    else
        graph.exec = nullptr;
    if (captured != nullptr) cudaGraphDestroy(captured);
    if (graph.single) cudaGetLastError();
    return !graph.single;
}

}  // namespace qb
