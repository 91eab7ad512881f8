// Pinned host staging for uploads: one process-wide pool per device, shared by the plans of that device.
//
// A copy from pageable memory makes the driver wait for the stream, bounce the data through its own pinned buffer
// and return only when that is done, so a batch bound from a NumPy array used to cost the step a drained GPU.
// Here the caller's array is copied into a pinned block at once (it may be reused when the call returns) and the
// transfer is queued on the stream; the block returns to the pool when its event has completed.
#pragma once
#include <cuda_runtime.h>

#include <cstddef>

namespace qb {

constexpr size_t STAGING_BLOCK_BYTES = (size_t)1 << 20;  // one transfer; larger arrays go in pieces, so that the
                                                         // host copy of one piece overlaps the transfer of the last
// A block costs 1 to 3 ms to page-lock and its transfer 0.03 ms: a plan's first inputs, which nothing runs ahead of, go
// through two blocks (a 16 MiB batch through sixteen new ones made the first bind of a plan 50 ms longer); later
// batches, queued behind steps still running, may take the pool to its bound.
constexpr int STAGING_FIRST_BLOCKS = 2;
constexpr int STAGING_BLOCKS = 16;                       // bound of the pool: 16 MiB of pinned memory per device

struct StagingBlock {
    unsigned char* host = nullptr;
    cudaEvent_t done = nullptr;
    bool queued = false;  // a transfer from it may still be running
};

// Users of the pool of `device` (the current device of the calling thread); the last one out frees the memory.
void staging_attach(int device);
void staging_detach(int device);
// A block no transfer is reading; while all have one, a new block up to `limit` of them, else the oldest after its transfer.
// *out is null when all blocks are in other callers' hands or no memory can be page-locked, and the caller then copies
// without staging.
cudaError_t staging_acquire(int device, int limit, StagingBlock** out);
// Transfers from `block` queued on `stream` so far must finish before it is handed out again.
cudaError_t staging_release(int device, StagingBlock* block, cudaStream_t stream);

}  // namespace qb
