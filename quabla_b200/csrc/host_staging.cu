// Pool of pinned staging blocks (see host_staging.h).
#include "host_staging.h"

#include <deque>
#include <memory>
#include <mutex>
#include <vector>

namespace qb {

namespace {

struct Pool {
    int users = 0;
    std::vector<std::unique_ptr<StagingBlock>> blocks;
    std::deque<StagingBlock*> idle;  // oldest transfer first
    void clear() {
        for (auto& b : blocks) {
            if (b->queued) cudaEventSynchronize(b->done);
            cudaEventDestroy(b->done);
            cudaFreeHost(b->host);
        }
        blocks.clear();
        idle.clear();
    }
};

std::mutex g_mutex;

Pool& pool(int device) {
    static std::vector<std::unique_ptr<Pool>>* pools = new std::vector<std::unique_ptr<Pool>>();  // never destroyed:
    while ((int)pools->size() <= device) pools->emplace_back(new Pool());  // plans may outlive static destructors
    return *(*pools)[device];
}

}  // namespace

void staging_attach(int device) {
    std::lock_guard<std::mutex> lock(g_mutex);
    ++pool(device).users;
}

void staging_detach(int device) {
    std::lock_guard<std::mutex> lock(g_mutex);
    Pool& p = pool(device);
    // Blocks handed out are back by now: a plan returns every block before its call ends.
    if (--p.users == 0) p.clear();
}

// Null when page-locked memory or an event is not to be had; no error is left pending.
static std::unique_ptr<StagingBlock> new_block() {
    std::unique_ptr<StagingBlock> fresh(new StagingBlock());
    void* raw = nullptr;
    if (cudaHostAlloc(&raw, STAGING_BLOCK_BYTES, cudaHostAllocPortable) == cudaSuccess) {
        if (cudaEventCreateWithFlags(&fresh->done, cudaEventDisableTiming) == cudaSuccess) {
            fresh->host = static_cast<unsigned char*>(raw);
            return fresh;
        }
        cudaFreeHost(raw);
    }
    cudaGetLastError();
    return nullptr;
}

cudaError_t staging_acquire(int device, int limit, StagingBlock** out) {
    *out = nullptr;
    StagingBlock* block = nullptr;
    {
        std::lock_guard<std::mutex> lock(g_mutex);
        Pool& p = pool(device);
        const bool oldest_done = !p.idle.empty() && (!p.idle.front()->queued || cudaEventQuery(p.idle.front()->done) == cudaSuccess);
        if (!oldest_done && (int)p.blocks.size() < (p.idle.empty() ? STAGING_BLOCKS : limit)) {
            if (std::unique_ptr<StagingBlock> fresh = new_block()) {
                *out = fresh.get();
                p.blocks.push_back(std::move(fresh));
                return cudaSuccess;
            }
        }
        if (p.idle.empty()) return cudaSuccess;  // none to be had, or all in other callers' hands at this instant
        block = p.idle.front();
        p.idle.pop_front();
    }
    *out = block;
    const cudaError_t e = block->queued ? cudaEventSynchronize(block->done) : cudaSuccess;
    block->queued = false;
    return e;
}

cudaError_t staging_release(int device, StagingBlock* block, cudaStream_t stream) {
    const cudaError_t e = cudaEventRecord(block->done, stream);
    block->queued = e == cudaSuccess;
    std::lock_guard<std::mutex> lock(g_mutex);
    pool(device).idle.push_back(block);
    return e;
}

}  // namespace qb
