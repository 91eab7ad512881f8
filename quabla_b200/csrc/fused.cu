// Instantiations of the fused engine.
#include "fused.h"

#include <algorithm>
#include <cstdlib>
#include <cstring>

#include "fused_kernel.cuh"
#include "fused_dmma_kernel.cuh"
#include "fused_mma_kernel.cuh"

namespace qb {

namespace {

template <int CODE>
FusedEntry<float> simt_entry() {
    typedef FusedGeom<CODE> G;
    FusedEntry<float> e;
    e.kernel = fused_step_kernel<CODE>;
    e.streams = G::S;
    e.tile_points = G::TP;
    e.smem_bytes = G::SMEM_BASE_BYTES;
    e.scratch_per_layer = G::SCRATCH_PER_CTA;
    e.tensor_core = false;
    e.dw_bytes = 0;
    e.width = G::W;
    e.threads = FUSED_THREADS;
    e.ctas_per_sm = 1;
    return e;
}

// QB200_FUSED=simt keeps the FP32-pipe variant for float32 width-64 networks (for comparisons); the default is the
// tensor-core variant.
bool want_simt() {
    const char* env = getenv("QB200_FUSED");
    return env != nullptr && strcmp(env, "simt") == 0;
}

}  // namespace

// Signature codes: 0 = value only; 1 = {1}; 2 = {2}; 3 = {3}; 4 = {4}; 6 = {1,1};
// 7 = {2,1}; 11 = {1,2}; 12 = {2,2}; SIG_MERGED + 6 / 31 = {1,1} / {1,1,1} plus the merged
// second-order stream (2-D / 3-D Laplacian).
#define QB_CASE(CODE)               \
    if (code == CODE) {             \
        *out = simt_entry<CODE>();  \
        return true;                \
    }

template <typename T>
static bool padded_lookup(int width, int layers, int code, int act, FusedEntry<T>* out) {
    if (width <= 16) return fused_mma_lookup<T, 16>(layers, code, act, out);
    if (width <= 32) return fused_mma_lookup<T, 32>(layers, code, act, out);
    if (width <= 48) return fused_mma_lookup<T, 48>(layers, code, act, out);
    if (width <= 64) return fused_mma_lookup<T, 64>(layers, code, act, out);
    return false;
}

template <>
bool fused_lookup<float>(int width, bool uniform, int layers, int code, int act, FusedEntry<float>* out) {
    if (act != ACT_TANH && act != ACT_SIN) return false;
    if (want_simt()) {
        if (width != 64 || !uniform || act != ACT_TANH) return false;
        QB_CASE(0) QB_CASE(1) QB_CASE(2) QB_CASE(4) QB_CASE(7) QB_CASE(12) QB_CASE(SIG_MERGED + 6)
        return false;
    }
    return padded_lookup<float>(width, layers, code, act, out);
}

template <>
bool fused_lookup<double>(int width, bool, int layers, int code, int act, FusedEntry<double>* out) {
    if (act != ACT_TANH && act != ACT_SIN) return false;
    return padded_lookup<double>(width, layers, code, act, out);
}

template <typename T>
cudaError_t fused_launch(const FusedEntry<T>& entry, int grid, size_t smem, cudaStream_t stream, const FusedArgs<T>& args) {
    // The bound of every launch, not of this one: plans of other depths share the kernel, and a thread that launches one
    // of them must not lower what another has just raised.
    cudaError_t e = cudaFuncSetAttribute(reinterpret_cast<const void*>(entry.kernel),
                                         cudaFuncAttributeMaxDynamicSharedMemorySize, (int)FUSED_MAX_SMEM);
    if (e != cudaSuccess) return e;
    if (entry.ctas_per_sm > 1) {
        // Co-residency needs the whole shared-memory carve-out.
        e = cudaFuncSetAttribute(reinterpret_cast<const void*>(entry.kernel),
                                 cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared);
        if (e != cudaSuccess) return e;
    }
    entry.kernel<<<grid, entry.threads, smem, stream>>>(args);
    return cudaGetLastError();
}

template <>
size_t fused_weight_image_bytes<float>(int hidden_to_hidden, int width) {
    return (size_t)std::max(hidden_to_hidden, 1) * 6 * width * (width + 8);
}
template <>
size_t fused_weight_image_bytes<double>(int hidden_to_hidden, int width) {
    return (size_t)std::max(hidden_to_hidden, 1) * 8 * width * (width + 4);
}

static PrepArgs prep_args(const int* w_off, const int* rows, const int* cols, int layers) {
    PrepArgs p;
    p.layers = layers;
    for (int i = 0; i <= FUSED_MAX_LAYERS; ++i) {
        p.w_off[i] = i < layers ? w_off[i] : 0;
        p.rows[i] = i < layers ? rows[i] : 0;
        p.cols[i] = i < layers ? cols[i] : 0;
    }
    return p;
}

template <>
cudaError_t fused_prep_launch<float>(const float* params, const int* w_off, const int* rows, const int* cols,
                                     int hidden_to_hidden, int width, void* images, cudaStream_t stream) {
    if (hidden_to_hidden < 1) return cudaSuccess;
    const PrepArgs p = prep_args(w_off, rows, cols, hidden_to_hidden);
    const dim3 grid(4, hidden_to_hidden);
    uint32_t* out = static_cast<uint32_t*>(images);
    if (width == 16) prep_weights_kernel<16><<<grid, 256, 0, stream>>>(params, p, out);
    if (width == 32) prep_weights_kernel<32><<<grid, 256, 0, stream>>>(params, p, out);
    if (width == 48) prep_weights_kernel<48><<<grid, 256, 0, stream>>>(params, p, out);
    if (width == 64) prep_weights_kernel<64><<<grid, 256, 0, stream>>>(params, p, out);
    return cudaGetLastError();
}
template <>
cudaError_t fused_prep_launch<double>(const double* params, const int* w_off, const int* rows, const int* cols,
                                      int hidden_to_hidden, int width, void* images, cudaStream_t stream) {
    if (hidden_to_hidden < 1) return cudaSuccess;
    prep_weights64_kernel<<<dim3(4, hidden_to_hidden), 256, 0, stream>>>(
        params, prep_args(w_off, rows, cols, hidden_to_hidden), width, static_cast<double*>(images));
    return cudaGetLastError();
}

// One thread waits, with a short poll limit, on a barrier that nothing ever completes: the wait
// gives up and raises *error exactly as a staged copy that never lands would.  Used by the host to
// exercise the error path of a plan without any faulting or endless kernel.
__global__ void unarmed_wait_kernel(int* error) {
    __shared__ uint64_t bar;
    if (threadIdx.x == 0) {
        mbar_init(&bar, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        mbar_wait_limited(&bar, 0u, error, 64);
    }
}

cudaError_t unarmed_wait_launch(int* error, cudaStream_t stream) {
    unarmed_wait_kernel<<<1, 32, 0, stream>>>(error);
    return cudaGetLastError();
}

template cudaError_t fused_launch<float>(const FusedEntry<float>&, int, size_t, cudaStream_t, const FusedArgs<float>&);
template cudaError_t fused_launch<double>(const FusedEntry<double>&, int, size_t, cudaStream_t, const FusedArgs<double>&);

}  // namespace qb
