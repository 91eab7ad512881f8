// Lookup of the fused-engine kernel instantiations (see fused_kernel.cuh).
#pragma once
#include <cuda_runtime.h>

#include <cstddef>

namespace qb {

template <typename T> struct FusedArgs;

template <typename T>
struct FusedEntry {
    void (*kernel)(FusedArgs<T>);
    int streams;                  // S
    int tile_points;              // TP
    size_t smem_bytes;            // dynamic shared memory per CTA, without the residual program
    size_t dw_bytes;              // tensor-core variant: running weight-gradient sums of one layer, in shared memory
                                  // behind the program when they fit, else in global memory
    size_t scratch_per_layer;     // saved-jet elements per CTA per hidden layer (each of Z and H)
    bool tensor_core;             // tensor-core variant: needs the weight images
    int width;                    // hidden width the kernel is built for (networks up to it run padded)
    int threads;                  // threads per CTA
    int ctas_per_sm;              // CTAs the kernel is sized to co-reside on one SM
};

constexpr size_t FUSED_MAX_SMEM = 227 * 1024;
constexpr size_t FUSED_SM_SMEM = 228 * 1024;      // of an SM; a resident CTA takes FUSED_CTA_SMEM of it besides its own
constexpr size_t FUSED_CTA_SMEM = 1024;

// Dynamic shared memory of a launch: the regions plus the staged residual program.
template <typename T>
inline size_t fused_smem_bytes(const FusedEntry<T>& entry, int n_instr) {
    return entry.smem_bytes + (size_t)n_instr * 16 + 16;
}

// True when a kernel exists for this dtype, largest hidden width, number of hidden layers, derivative signature code
// (sum over directions j of order_j * 5^j) and activation (ACT_TANH or ACT_SIN).  `uniform`: every hidden layer has
// that width (the FP32-pipe kernels have no padding).
template <typename T>
bool fused_lookup(int width, bool uniform, int layers, int code, int act, FusedEntry<T>* out);

// Tensor-core kernels of one padded width (fused_mma_w*.cu, fused_dmma_w*.cu).
template <typename T, int W>
bool fused_mma_lookup(int layers, int code, int act, FusedEntry<T>* out);

// Launches entry.kernel with `smem` bytes of dynamic shared memory.
template <typename T>
cudaError_t fused_launch(const FusedEntry<T>& entry, int grid, size_t smem, cudaStream_t stream, const FusedArgs<T>& args);

// Bytes of the weight images of `hidden_to_hidden` layers padded to `width`.
template <typename T>
size_t fused_weight_image_bytes(int hidden_to_hidden, int width);
// Writes the images from the flat parameters; image i is network layer 1 + i, of
// rows[i] x cols[i] at offset w_off[i].
template <typename T>
cudaError_t fused_prep_launch(const T* params, const int* w_off, const int* rows, const int* cols, int hidden_to_hidden,
                              int width, void* images, cudaStream_t stream);
// One thread's bounded wait on a barrier that is never completed: raises *error when it gives up.
cudaError_t unarmed_wait_launch(int* error, cudaStream_t stream);

}  // namespace qb
