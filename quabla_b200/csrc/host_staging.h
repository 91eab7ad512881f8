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
constexpr int STAGING_BLOCKS = 16;                       // bound of the pool: 16 MiB of pinned memory per device

struct StagingBlock {
    unsigned char* host = nullptr;
    cudaEvent_t done = nullptr;
    bool queued = false;  // a transfer from it may still be running
};

// Users of the pool of `device` (the current device of the calling thread); the last one out frees the memory.
void staging_attach(int device);
void staging_detach(int device);
// A block no transfer is reading (waits for the oldest transfer when every block has one); *out is null when all
// blocks are in other callers' hands, and the caller then copies without staging.
cudaError_t staging_acquire(int device, StagingBlock** out);
// Transfers from `block` queued on `stream` so far must finish before it is handed out again.
cudaError_t staging_release(int device, StagingBlock* block, cudaStream_t stream);

}  // namespace qb
