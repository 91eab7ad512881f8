// Entries of the tensor-core fused kernels of one padded hidden width; every fused_mma_w*.cu instantiates one width.
#pragma once
#include "fused.h"
#include "fused_dmma_kernel.cuh"
#include "fused_mma_kernel.cuh"

namespace qb {

template <typename T, typename G>
FusedEntry<T> mma_entry_of(void (*kernel)(FusedArgs<T>), int layers) {
    FusedEntry<T> e;
    e.kernel = kernel;
    e.streams = G::S;
    e.tile_points = G::TP;
    e.smem_bytes = G::base_bytes(layers);
    e.dw_bytes = G::DW_BYTES;
    e.scratch_per_layer = G::SCRATCH_PER_CTA;
    e.tensor_core = true;
    e.width = G::W;
    e.threads = G::THREADS;
    e.ctas_per_sm = G::MIN_CTAS;
    return e;
}

// Signature codes as in fused.cu.
#define QB_MMA_CASE(T, W, CODE, GEOM, KERNEL)                                                                             \
    if (code == CODE) {                                                                                                  \
        *out = act == ACT_TANH ? mma_entry_of<T, GEOM<CODE, W>>(KERNEL<CODE, W, ACT_TANH>, layers)                        \
                               : mma_entry_of<T, GEOM<CODE, W>>(KERNEL<CODE, W, ACT_SIN>, layers);                        \
        return true;                                                                                                     \
    }
#define QB_MMA_LOOKUP(T, W, GEOM, KERNEL)                                                                                 \
    template <>                                                                                                          \
    bool fused_mma_lookup<T, W>(int layers, int code, int act, FusedEntry<T>* out) {                                     \
        QB_MMA_CASE(T, W, 0, GEOM, KERNEL) QB_MMA_CASE(T, W, 1, GEOM, KERNEL) QB_MMA_CASE(T, W, 2, GEOM, KERNEL)          \
        QB_MMA_CASE(T, W, 4, GEOM, KERNEL) QB_MMA_CASE(T, W, 7, GEOM, KERNEL) QB_MMA_CASE(T, W, 12, GEOM, KERNEL)         \
        QB_MMA_CASE(T, W, SIG_MERGED + 6, GEOM, KERNEL) QB_MMA_CASE(T, W, SIG_MERGED + 31, GEOM, KERNEL)                  \
        QB_MMA_CASE(T, W, SIG_MERGED + 156, GEOM, KERNEL)                                                                 \
        return false;                                                                                                    \
    }

}  // namespace qb
