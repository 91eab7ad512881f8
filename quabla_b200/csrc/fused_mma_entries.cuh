// Entries of the split-operand fused kernels of one padded hidden width; every fused_mma_w*.cu instantiates one width.
#pragma once
#include "fused.h"
#include "fused_mma_kernel.cuh"

namespace qb {

template <int CODE, int W, int ACT>
FusedEntry<float> make_mma_entry(int layers) {
    typedef MmaGeom<CODE, W> G;
    FusedEntry<float> e;
    e.kernel = fused_mma_kernel<CODE, W, ACT>;
    e.streams = G::S;
    e.tile_points = G::TP;
    e.smem_bytes = G::base_bytes(layers);
    e.dw_bytes = G::DW_BYTES;
    e.scratch_per_layer = G::SCRATCH_PER_CTA;
    e.tensor_core = true;
    e.width = W;
    e.threads = G::THREADS;
    e.ctas_per_sm = G::MIN_CTAS;
    return e;
}

// Signature codes as in fused.cu.
#define QB_MMA_CASE(W, CODE)                                                                                             \
    if (code == CODE) {                                                                                                  \
        *out = act == ACT_TANH ? make_mma_entry<CODE, W, ACT_TANH>(layers) : make_mma_entry<CODE, W, ACT_SIN>(layers);   \
        return true;                                                                                                     \
    }
#define QB_MMA_LOOKUP(W)                                                                                                 \
    template <>                                                                                                          \
    bool fused_mma_lookup<W>(int layers, int code, int act, FusedEntry<float>* out) {                                    \
        QB_MMA_CASE(W, 0) QB_MMA_CASE(W, 1) QB_MMA_CASE(W, 2) QB_MMA_CASE(W, 4) QB_MMA_CASE(W, 7) QB_MMA_CASE(W, 12)     \
        QB_MMA_CASE(W, SIG_MERGED + 6) QB_MMA_CASE(W, SIG_MERGED + 31) QB_MMA_CASE(W, SIG_MERGED + 156)                  \
        return false;                                                                                                    \
    }

}  // namespace qb
