// Host side of the tcgen05 float32 GEMMs.
#include "tc_gemm.h"

#include <cstdlib>
#include <cstring>

#include "tc_tma_gemm.cuh"

namespace qb {

static bool tc_switch_on() {
    const char* env = getenv("QB200_TC");
    return !(env != nullptr && strcmp(env, "0") == 0);
}

// How the forward and data-gradient GEMMs split their float32 operands (tc_tma_gemm.cuh): two float16 parts of scaled
// rows at every size; it is both the fastest (six tensor instructions and 32 KB of loads per k-tile against eight and
// 48 KB, and twelve and 48 KB) and the most accurate of the three.  QB200_TC_COR=tf32 or =bf16 (read at every call)
// selects one of the others for comparisons: three tf32 products, or tf32 with bfloat16 corrections.
TcScheme tc_scheme() {
    const char* env = getenv("QB200_TC_COR");
    if (env != nullptr && strcmp(env, "tf32") == 0) return TC_TF32;
    if (env != nullptr && strcmp(env, "bf16") == 0) return TC_BF16;
    return TC_F16;
}

bool tc_rows_ok(int N, int K) { return N % 64 == 0 && N >= 64 && N <= 256 && K % TC_BK == 0 && K >= TC_BK; }

bool tc_wgrad_ok(int Mw, int N) { return Mw % TC_BM == 0 && N % 64 == 0 && N >= 64 && N <= 256; }

size_t tc_image_words(int K, int N) { return (size_t)4 * K * N; }

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

static EncodeTiledFn encode_tiled() {
    static EncodeTiledFn fn = [] {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult status;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &status) != cudaSuccess ||
            status != cudaDriverEntryPointSuccess)
            p = nullptr;
        return reinterpret_cast<EncodeTiledFn>(p);
    }();
    return fn;
}

bool tc_available() {
    static const bool available = tc_switch_on() && encode_tiled() != nullptr;
    return available;
}

// Row-major float32 matrix [rows][cols] with leading dimension ld, boxes of box_cols x box_rows,
// the given 128-byte swizzle, zero fill outside the matrix.
static bool make_map(CUtensorMap* map, const float* base, long long rows, int cols, int ld, int box_cols, int box_rows,
                     CUtensorMapSwizzle swizzle) {
    const cuuint64_t dims[2] = {(cuuint64_t)cols, (cuuint64_t)rows};
    const cuuint64_t strides[1] = {(cuuint64_t)ld * sizeof(float)};
    const cuuint32_t box[2] = {(cuuint32_t)box_cols, (cuuint32_t)box_rows};
    const cuuint32_t elem[2] = {1, 1};
    return encode_tiled()(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, const_cast<float*>(base), dims, strides, box, elem,
                          CU_TENSOR_MAP_INTERLEAVE_NONE, swizzle, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                          CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// 16-bit pair matrix of tc2_prepare_launch: [rows][2 * inner] halves, boxes of 64 halves (128 bytes) x box_rows under
// the 128-byte swizzle.
static bool make_map16(CUtensorMap* map, const void* base, long long rows, int inner, int box_rows) {
    const cuuint64_t dims[2] = {(cuuint64_t)(2 * inner), (cuuint64_t)rows};
    const cuuint64_t strides[1] = {(cuuint64_t)(2 * inner) * 2};
    const cuuint32_t box[2] = {64, (cuuint32_t)box_rows};
    const cuuint32_t elem[2] = {1, 1};
    return encode_tiled()(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(base), dims, strides, box, elem,
                          CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                          CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

TcImage tc_image(float* words, int K, int N) {
    const size_t kn = (size_t)K * N;
    TcImage im;
    im.first = words;
    im.second = words + kn;
    im.third = words + 2 * kn;
    im.fourth = words + 3 * kn;
    return im;
}

cudaError_t tc2_prepare_launch(const float* w, int K, int N, float* words, TcScheme scheme, cudaStream_t stream) {
    const TcImage im = tc_image(words, K, N);
    const dim3 tiles((N + 31) / 32, (K + 31) / 32), block(32, 8);
    if (scheme == TC_F16)
        t2_prepare_f16_kernel<<<(N + K + 7) / 8, 256, 0, stream>>>(w, K, N, reinterpret_cast<__half*>(im.first),
                                                                    reinterpret_cast<__half*>(im.second), im.third, im.third + N);
    else if (scheme == TC_BF16)
        t2_prepare16_kernel<<<tiles, block, 0, stream>>>(w, K, N, im.first, reinterpret_cast<uint16_t*>(im.second),
                                                         reinterpret_cast<uint16_t*>(im.third), im.fourth);
    else
        t2_prepare_kernel<<<tiles, block, 0, stream>>>(w, K, N, im.first, reinterpret_cast<uint32_t*>(im.second),
                                                       reinterpret_cast<uint32_t*>(im.third));
    return cudaGetLastError();
}

template <bool WGRAD, int BN, bool PRELO, bool C16 = false, bool F16 = false>
static cudaError_t launch2(const CUtensorMap& ma, const CUtensorMap& mb, const CUtensorMap& mblo, const CUtensorMap& mc,
                           const TcTmaArgs& a, dim3 grid, cudaStream_t stream) {
    typedef T2Geom<WGRAD, BN, PRELO, C16, F16> G;
    cudaError_t e = cudaFuncSetAttribute(reinterpret_cast<const void*>(tc_tma_gemm_kernel<WGRAD, BN, PRELO, C16, F16>),
                                         cudaFuncAttributeMaxDynamicSharedMemorySize, G::SMEM_BYTES);
    if (e != cudaSuccess) return e;
    tc_tma_gemm_kernel<WGRAD, BN, PRELO, C16, F16><<<grid, T2_THREADS_TOTAL, G::SMEM_BYTES, stream>>>(ma, mb, mblo, mc, a);
    return cudaGetLastError();
}

cudaError_t tc2_rows_launch(const float* A, int M, int K_w, int N_w, const float* w, float* words, bool dgrad, float* C,
                            const float* bias, int bias_rows, TcScheme scheme, int* error, cudaStream_t stream) {
    const int N = dgrad ? K_w : N_w, K = dgrad ? N_w : K_w;
    const int BN = N % 128 == 0 ? 128 : 64;
    const TcImage im = tc_image(words, K_w, N_w);
    // Bt and its second matrix; F16 has the pair matrix alone.
    const float* pair = scheme == TC_F16 ? (dgrad ? im.second : im.first) : (dgrad ? im.third : im.second);
    const float* Bt = scheme == TC_F16 ? pair : !dgrad ? im.first : scheme == TC_BF16 ? im.fourth : w;
    CUtensorMap ma, mb, mblo, mc;
    if (!make_map(&ma, A, M, K, K, T2_BK, T2_BM, CU_TENSOR_MAP_SWIZZLE_128B) ||
        !make_map(&mb, Bt, N, K, K, T2_BK, BN, CU_TENSOR_MAP_SWIZZLE_128B) ||
        !(scheme == TC_TF32 ? make_map(&mblo, pair, N, K, K, T2_BK, BN, CU_TENSOR_MAP_SWIZZLE_128B)
                            : make_map16(&mblo, pair, N, K, BN)) ||
        !make_map(&mc, C, M, N, N, 32, T2_BM, CU_TENSOR_MAP_SWIZZLE_128B))
        return cudaErrorInvalidValue;
    TcTmaArgs a;
    memset(&a, 0, sizeof(a));
    a.C = C;
    a.bias = bias;
    a.M = M;
    a.N = N;
    a.K = K;
    a.ldc = N;
    a.bias_rows = bias_rows;
    a.units = ((M + T2_BM - 1) / T2_BM) * (N / BN);
    a.scale = im.third + (dgrad ? N_w : 0);
    a.error = error;
    const dim3 grid(a.units < 148 ? a.units : 148);
    if (scheme == TC_F16)
        return BN == 128 ? launch2<false, 128, true, false, true>(ma, mb, mblo, mc, a, grid, stream)
                         : launch2<false, 64, true, false, true>(ma, mb, mblo, mc, a, grid, stream);
    if (scheme == TC_BF16)
        return BN == 128 ? launch2<false, 128, true, true>(ma, mb, mblo, mc, a, grid, stream)
                         : launch2<false, 64, true, true>(ma, mb, mblo, mc, a, grid, stream);
    return BN == 128 ? launch2<false, 128, true>(ma, mb, mblo, mc, a, grid, stream)
                     : launch2<false, 64, true>(ma, mb, mblo, mc, a, grid, stream);
}

cudaError_t tc2_wgrad_launch(const float* H, int ldh, const float* G, int ldg, float* partials, int rows, int Mw, int N,
                             int rows_per_slice, int* error, cudaStream_t stream) {
    const int BN = N % 128 == 0 ? 128 : 64;
    const int slices = (rows + rows_per_slice - 1) / rows_per_slice;
    CUtensorMap ma, mb, mc;
    if (!make_map(&ma, H, rows, Mw, ldh, 32, T2_BK, CU_TENSOR_MAP_SWIZZLE_128B_ATOM_32B) ||
        !make_map(&mb, G, rows, N, ldg, 32, T2_BK, CU_TENSOR_MAP_SWIZZLE_128B_ATOM_32B) ||
        !make_map(&mc, partials, (long long)slices * Mw, N, N, 32, T2_BM, CU_TENSOR_MAP_SWIZZLE_128B))
        return cudaErrorInvalidValue;
    TcTmaArgs a;
    memset(&a, 0, sizeof(a));
    a.C = partials;
    a.M = Mw;
    a.N = N;
    a.K = rows;
    a.ldc = N;
    a.k_slice = rows_per_slice;
    a.error = error;
    const dim3 grid(Mw / T2_BM, N / BN, slices);  // the tiles of one slice run together and share its rows in L2
    return BN == 128 ? launch2<true, 128, false>(ma, mb, mb, mc, a, grid, stream)
                     : launch2<true, 64, false>(ma, mb, mb, mc, a, grid, stream);
}

}  // namespace qb
