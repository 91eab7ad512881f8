// Fused engine, float32, hidden widths up to 64, weight contractions on the tensor cores with operands split into
// two float16 parts.
//
// Split.  A block of 16 x 16 elements (16 points x 16 units of one stream) is scaled by a power of two so that its
// largest element lies in [2^13, 2^14), and every scaled element y is written as hi + lo with hi = f16(y) and
// lo = f16(y - hi).  The pair carries y to 2^-23 of itself down to 2^-16 of the block's largest element and to
// 2^-39 of that largest element below (hi and lo are then subnormal).  A product A.B is lo.hi + hi.lo + hi.hi,
// three m16n8k16 instructions per 16 contraction elements: half the tensor-pipe time and half the instructions of three
// tf32 products, which left 2e-7 per product against 1e-7 here (the dropped lo.lo is of random sign).  One
// contraction step of 16 reads exactly one block of either operand, so the blocks' scales multiply the step's
// partial sum on its way into the running sum: a multiply-add where a plain addition was needed anyway.
//
// Same structure as fused_step_kernel (fused_kernel.cuh): persistent CTAs walk tiles of 16 points, run forward /
// residual / reverse sweep per tile, keep the saved jets in an L2-resident per-CTA scratch and accumulate weight
// gradients per CTA.  Warp w owns units 16 w .. 16 w + 15 (W / 16 warps): for every stream the 16 x 16 tile
// (points x units) as two m16n8 accumulator fragments, so thread (g = lane / 4, t = lane % 4) holds points
// {g, g + 8} x units {2t, 2t + 1} of both fragments for ALL streams, and the jet composition stays register-only.
// Networks narrower than W (or of unequal widths) run padded with zero weights: a padded unit's activation meets
// only zero weights and its cotangent is zero.
//
// Bound: issue slots and latencies of the epilogues between the contractions (the tensor pipe is not the limit), which
// is why a CTA is one point group with as few registers as its stream count allows: as many CTAs as fit
// overlap one another's phases (three per SM at width 64 and up to four streams).
// Measured against the 3xTF32 kernel before it: 65,536-point 2-D Poisson interior 590 -> 330 us, 1,048,576-point beam step
// 11.15 -> 7.24 ms, width 50 at 20,000 points 845 -> 150 us per step (layer by layer before).
//
// Replaces the reference's per-node plan execution (crates/quabla-core/src/tensor_ir/cuda.rs:1792-2972) and its
// cuBLAS strided-batched GEMV-shaped calls (cuda.rs:4936-5035).
#pragma once
#include <cuda_fp16.h>

#include <cstdint>
#include <cstdio>

#include "fused_kernel.cuh"

namespace qb {

// Four 8x8 matrices of 16-bit elements; thread (g, t) receives elements 2t, 2t + 1 of row g of each (TRANS: of
// column g), the m16n8k16 fragment layouts.
template <bool TRANS>
__device__ __forceinline__ void ldmatrix_x4(uint32_t (&r)[4], const __half* row_ptr) {
    const uint32_t at = (uint32_t)__cvta_generic_to_shared(row_ptr);
    if (TRANS)
        asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
                     : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                     : "r"(at));
    else
        asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
                     : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                     : "r"(at));
}

// d += a (16x16, row) * b (16x8, col), float16 operands, float32 accumulate.  Not volatile: the accumulator operands
// carry the dependencies, the compiler may interleave independent chains.
__device__ __forceinline__ void mma_f16(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

// acc += f * (A_lo.B_hi + A_hi.B_lo + A_hi.B_hi) of one 16 x 16 by 16 x 16 step.  The tensor core adds into its
// accumulator with truncation, so every step chains its three products from zero and the partial is added to the
// running sum with a round-to-nearest multiply-add.
__device__ __forceinline__ void mma_step(float (&acc)[2][4], const uint32_t (&ahi)[4], const uint32_t (&alo)[4],
                                         const uint32_t (&bhi)[4], const uint32_t (&blo)[4], float f) {
#pragma unroll
    for (int j = 0; j < 2; ++j) {
        float part[4] = {0.0f, 0.0f, 0.0f, 0.0f};
        mma_f16(part, alo, bhi[2 * j], bhi[2 * j + 1]);
        mma_f16(part, ahi, blo[2 * j], blo[2 * j + 1]);
        mma_f16(part, ahi, bhi[2 * j], bhi[2 * j + 1]);
#pragma unroll
        for (int c = 0; c < 4; ++c) acc[j][c] = fmaf(part[c], f, acc[j][c]);
    }
}

// Power-of-two scale of a block whose largest magnitude has the bit pattern `largest`: *inverse maps it into
// [2^13, 2^14), the returned factor maps back.  Blocks below 2^-113 (and empty ones) share the scale of that size.
__device__ __forceinline__ float block_scale(uint32_t largest, float* inverse) {
    const uint32_t e = max(largest >> 23, 14u);
    *inverse = __uint_as_float((267u - e) << 23);
    return __uint_as_float((e - 13u) << 23);
}

// Mean relative loss of mma_step's truncating accumulations: a factor common to all contractions, which neither the
// number of points nor of terms averages out, so it is put back where that costs nothing: into the weights' lo parts and
// into the finished weight-gradient sums.  Measured as <error, exact> / <exact, exact> of 40,000 16 x 16 x 16 steps against float64:
// -3.9e-8 (normal operands), -4.1e-8 (uniform), -4.4e-8 (positive).  Without it gradients of networks of width 16, 32 and
// 50 were 2 to 5 times further from float64 than plain float32 multiply-adds.
constexpr float MMA_TRUNCATION = 4.1e-8f;

// Two scaled elements as packed float16 hi and lo pairs, raised by `gain` of themselves.
__device__ __forceinline__ void split_f16(float x0, float x1, float inverse, uint32_t& hi, uint32_t& lo, float gain = 0.0f) {
    const float y0 = x0 * inverse, y1 = x1 * inverse;
    const __half2 h = __floats2half2_rn(y0, y1);
    const float2 back = __half22float2(h);
    const __half2 l = gain == 0.0f ? __floats2half2_rn(y0 - back.x, y1 - back.y)
                                   : __floats2half2_rn(fmaf(y0, gain, y0 - back.x), fmaf(y1, gain, y1 - back.y));
    hi = *reinterpret_cast<const uint32_t*>(&h);
    lo = *reinterpret_cast<const uint32_t*>(&l);
}

// ---- asynchronous staging: bulk copies (TMA engine, no multicast) and cp.async ----
__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void mbar_init(uint64_t* bar, int count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count));
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}
// Bulk copy global -> shared of `bytes` (multiple of 16, both addresses 16-byte aligned),
// completion counted on `bar`.
__device__ __forceinline__ void bulk_load(void* dst, const void* src, uint32_t bytes, uint64_t* bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                     smem_u32(dst)),
                 "l"(src), "r"(bytes), "r"(smem_u32(bar))
                 : "memory");
}
// Waits for phase `parity` of `bar`; gives up after a bounded number of polls and
// reports through *error (the kernel then finishes with wrong numbers, flagged).
__device__ __forceinline__ void mbar_wait_limited(uint64_t* bar, uint32_t parity, int* error, int limit) {
    uint32_t done = 0;
    for (int spin = 0; spin < limit && !done; ++spin) {
        asm volatile(
            "{ .reg .pred p; mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2; selp.u32 %0, 1, 0, p; }"
            : "=r"(done)
            : "r"(smem_u32(bar)), "r"(parity)
            : "memory");
    }
    if (!done) *error = 1;
}
__device__ __forceinline__ void mbar_wait(uint64_t* bar, uint32_t parity, int* error) {
    mbar_wait_limited(bar, parity, error, 1 << 22);
}
__device__ __forceinline__ void cp_async16(void* dst, const void* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_group 0;" ::: "memory"); }


// Weight images written by prep_weights_kernel, one per hidden-to-hidden layer: {hi, lo} planes [W][W + 8] halves of
// the row-major [in][out] matrix, zero-padded to W x W, scaled as one block; its factor goes to scales[layer].  The
// forward contraction reads it transposed (ldmatrix .trans), the data gradient as it is.
struct PrepArgs {
    int layers;                       // hidden-to-hidden layers
    int w_off[FUSED_MAX_LAYERS + 1];  // parameter offset of network layer 1 + i
    int rows[FUSED_MAX_LAYERS + 1];   // its true input and output widths
    int cols[FUSED_MAX_LAYERS + 1];
};

static __global__ void __launch_bounds__(1024) prep_weights_kernel(const float* __restrict__ params, PrepArgs p, int W,
                                                                   uint32_t* __restrict__ images, float* __restrict__ scales) {
    __shared__ uint32_t warp_max[32];
    const int layer = blockIdx.x, rows = p.rows[layer], cols = p.cols[layer];
    const float* w = params + p.w_off[layer];
    uint32_t largest = 0;
    for (int e = threadIdx.x; e < rows * cols; e += blockDim.x) largest = max(largest, __float_as_uint(w[e]) & 0x7fffffffu);
    largest = __reduce_max_sync(0xffffffffu, largest);
    if ((threadIdx.x & 31) == 0) warp_max[threadIdx.x >> 5] = largest;
    __syncthreads();
    largest = __reduce_max_sync(0xffffffffu, (threadIdx.x & 31) < (blockDim.x >> 5) ? warp_max[threadIdx.x & 31] : 0u);
    float inverse;
    const float scale = block_scale(largest, &inverse);
    if (threadIdx.x == 0) scales[layer] = scale;
    const int pairs = W / 2, stride = (W + 8) / 2, plane = W * stride;  // in 32-bit words
    uint32_t* img = images + (size_t)layer * 2 * plane;
    for (int e = threadIdx.x; e < W * pairs; e += blockDim.x) {
        const int r = e / pairs, c = 2 * (e % pairs);
        const float x0 = (r < rows && c < cols) ? w[r * cols + c] : 0.0f;
        const float x1 = (r < rows && c + 1 < cols) ? w[r * cols + c + 1] : 0.0f;
        uint32_t hi, lo;
        split_f16(x0, x1, inverse, hi, lo, MMA_TRUNCATION);
        img[r * stride + c / 2] = hi;
        img[plane + r * stride + c / 2] = lo;
    }
}

template <int CODE, int W_>
struct MmaGeom {
    typedef Sig<CODE> sig;
    static constexpr int W = W_;
    static constexpr int S = sig::S;
    static constexpr int NW = W / 16;            // warps = column blocks
    static constexpr int THREADS = 32 * NW;
    static constexpr int TP = 16;
    static constexpr int ROWS = S * TP;
    // Rows of W + 8 halves: 16-byte aligned, and the eight row addresses of an ldmatrix tile fall into distinct
    // bank groups for every W used (stride 4 (mod 8) words).
    static constexpr int LD = W + 8;
    static constexpr int PLANE = ROWS * LD;      // halves per operand plane
    static constexpr int WPLANE = W * LD;        // halves per weight plane
    static constexpr int ACT_BYTES = 4 * PLANE;  // hi and lo
    static constexpr int WIMG_BYTES = 4 * WPLANE;
    static constexpr int OFF_ACT = 0;                      // activations / cotangents, [hi, lo][ROWS][LD]
    static constexpr int OFF_HT = OFF_ACT + ACT_BYTES;     // previous layer's jets (weight-gradient operand), same layout
    static constexpr int OFF_WB = OFF_HT + ACT_BYTES;      // weight image of the contraction at hand
    static constexpr int OFF_RED = OFF_WB + WIMG_BYTES;    // [NW][S][TP] output-layer partials
    static constexpr int OFF_U = OFF_RED + 4 * NW * ROWS;  // [S][TP]
    static constexpr int OFF_UH = OFF_U + 4 * ROWS;        // [S][TP]
    static constexpr int OFF_BAR = OFF_UH + 4 * ROWS;      // two mbarriers
    static constexpr int OFF_VAR = OFF_BAR + 16;           // regions that depend on the depth:
    // block scales [L + 1][S][NW], weight scales [L], parameters {biases [L][W], first layer [4][W], output layer
    // [W]}, gradient sums of the same, of the output bias
    static __host__ __device__ constexpr size_t var_bytes(int L) {
        return 4 * ((size_t)(L + 1) * S * NW + L + 2 * (size_t)(L + 5) * W + 4);
    }
    static __host__ __device__ constexpr size_t base_bytes(int L) { return ((size_t)OFF_VAR + var_bytes(L) + 15) / 16 * 16; }
    static constexpr size_t DW_BYTES = 4 * (size_t)W * W;  // running weight-gradient sums of one layer
    // Registers decide how many CTAs share an SM: 168 per thread hold up to four streams, 224 to 255 more.
    static constexpr int MIN_CTAS = (S <= 4 ? 12 : 8) / NW;
    // Saved jets: the operand planes as they sit in shared memory, one bulk copy per layer.  Saved pre-activations:
    // read back by the thread that wrote them, so laid out per thread.
    static constexpr size_t SCRATCH_PER_CTA = (size_t)ROWS * LD;
};

// Optional per-phase cycle counters of CTA 0 (compile with -DQB_PHASE_TIMING), printed once per launch.
#ifdef QB_PHASE_TIMING
#define QB_PHASE(i)                                      \
    do {                                                 \
        if (tid == 0) {                                  \
            const long long now_ = clock64();            \
            phase_[i] += now_ - last_;                   \
            last_ = now_;                                \
        }                                                \
    } while (0)
#else
#define QB_PHASE(i)
#endif

// The warp's 16 x 16 block of every stream as scaled float16 pairs into the operand planes; scales [S][NW].
template <int S, int NW, int LD, int PLANE>
__device__ __forceinline__ void store_blocks(const float (&acc)[S][2][4], __half* planes, float* scales, int warp, int g, int t) {
    uint32_t largest[S];
#pragma unroll
    for (int s = 0; s < S; ++s) {
        uint32_t m = 0;
#pragma unroll
        for (int j = 0; j < 2; ++j)
#pragma unroll
            for (int c = 0; c < 4; ++c) m = max(m, __float_as_uint(acc[s][j][c]) & 0x7fffffffu);
        largest[s] = __reduce_max_sync(0xffffffffu, m);
    }
    uint32_t* words = reinterpret_cast<uint32_t*>(planes) + (g * LD + 16 * warp + 2 * t) / 2;
#pragma unroll
    for (int s = 0; s < S; ++s) {
        float inverse;
        const float scale = block_scale(largest[s], &inverse);
        if (g == 0 && t == 0) scales[s * NW + warp] = scale;
#pragma unroll
        for (int j = 0; j < 2; ++j)
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                uint32_t hi, lo;
                split_f16(acc[s][j][2 * i], acc[s][j][2 * i + 1], inverse, hi, lo);
                uint32_t* at = words + ((s * 16 + 8 * i) * LD + 8 * j) / 2;
                at[0] = hi;
                at[PLANE / 2] = lo;
            }
    }
}

// acc[s] = A[rows of stream s][W] * B[W][16 columns of this warp].  FORWARD: B(k, n) = W[k][n]; else B(k, n) = W[n][k].
template <int S, int NW, int LD, int PLANE, int WPLANE, bool FORWARD>
__device__ __forceinline__ void warp_contract(const __half* __restrict__ A, const __half* __restrict__ Wimg,
                                              const float* __restrict__ scales, float wscale, int warp, int lane,
                                              float (&acc)[S][2][4]) {
#pragma unroll
    for (int s = 0; s < S; ++s)
#pragma unroll
        for (int j = 0; j < 2; ++j)
#pragma unroll
            for (int c = 0; c < 4; ++c) acc[s][j][c] = 0.0f;
    const int mi = lane >> 3, rr = lane & 7;
    const __half* a_lane = A + (rr + (mi & 1) * 8) * LD + (mi >> 1) * 8;
    const __half* b_lane = FORWARD ? Wimg + ((mi & 1) * 8 + rr) * LD + 16 * warp + (mi >> 1) * 8
                                   : Wimg + (16 * warp + (mi >> 1) * 8 + rr) * LD + (mi & 1) * 8;
#pragma unroll
    for (int kb = 0; kb < NW; ++kb) {
        uint32_t bhi[4], blo[4];
        const __half* b = b_lane + (FORWARD ? kb * 16 * LD : kb * 16);
        ldmatrix_x4<FORWARD>(bhi, b);
        ldmatrix_x4<FORWARD>(blo, b + WPLANE);
#pragma unroll
        for (int s = 0; s < S; ++s) {
            uint32_t ahi[4], alo[4];
            ldmatrix_x4<false>(ahi, a_lane + s * 16 * LD + kb * 16);
            ldmatrix_x4<false>(alo, a_lane + s * 16 * LD + kb * 16 + PLANE);
            mma_step(acc[s], ahi, alo, bhi, blo, scales[s * NW + kb] * wscale);
        }
    }
}

// Column sums over the 16 points of the warp's block (v: this thread's four units, its two points already added);
// lanes with g == 0 add them to dst, which only this warp touches.
__device__ __forceinline__ void add_column_sums(float (&v)[4], float* dst, int lane, int col0, int t) {
#pragma unroll
    for (int c = 0; c < 4; ++c) {
        v[c] += __shfl_xor_sync(0xffffffffu, v[c], 4);
        v[c] += __shfl_xor_sync(0xffffffffu, v[c], 8);
        v[c] += __shfl_xor_sync(0xffffffffu, v[c], 16);
    }
    if (lane < 4) {
        dst[col0 + 2 * t] += v[0];
        dst[col0 + 2 * t + 1] += v[1];
        dst[col0 + 8 + 2 * t] += v[2];
        dst[col0 + 8 + 2 * t + 1] += v[3];
    }
}

template <int CODE, int W, int ACT>
__global__ void __launch_bounds__(MmaGeom<CODE, W>::THREADS, MmaGeom<CODE, W>::MIN_CTAS) fused_mma_kernel(FusedArgs<float> a) {
    typedef MmaGeom<CODE, W> G;
    typedef Sig<CODE> SG;
    constexpr int THREADS = G::THREADS, NW = G::NW, S = G::S, TP = G::TP, LD = G::LD, PLANE = G::PLANE, WPLANE = G::WPLANE;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __half* act = reinterpret_cast<__half*>(smem_raw + G::OFF_ACT);
    __half* ht = reinterpret_cast<__half*>(smem_raw + G::OFF_HT);
    __half* wbuf = reinterpret_cast<__half*>(smem_raw + G::OFF_WB);
    float* red = reinterpret_cast<float*>(smem_raw + G::OFF_RED);
    float* us = reinterpret_cast<float*>(smem_raw + G::OFF_U);
    float* uh = reinterpret_cast<float*>(smem_raw + G::OFF_UH);
    uint64_t* wbar = reinterpret_cast<uint64_t*>(smem_raw + G::OFF_BAR);  // weight image landed
    uint64_t* hbar = wbar + 1;                                            // saved jets landed
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int g = lane >> 2, t = lane & 3;
    const int col0 = warp * 16;  // first unit of the warp
    const int L = a.L, d0 = a.d0, HL = L - 1;
    const bool backward = a.forward_only == 0;
    float* scl = reinterpret_cast<float*>(smem_raw + G::OFF_VAR);  // [L][S][NW] activations, then one row for the cotangents
    float* scl_z = scl + L * S * NW;
    float* wscl = scl_z + S * NW;        // [L], by hidden-to-hidden layer
    float* pbias = wscl + L;             // [L][W]
    float* pfirst = pbias + L * W;       // [4][W]
    float* phead = pfirst + 4 * W;       // [W]
    float* gbias = phead + W;            // gradient sums in the same order
    float* gfirst = gbias + L * W;
    float* ghead = gfirst + 4 * W;
    int4* code = reinterpret_cast<int4*>(smem_raw + G::base_bytes(L));
    float* sz = a.scratch_z + (size_t)blockIdx.x * L * G::SCRATCH_PER_CTA;
    float* sh = a.scratch_h + (size_t)blockIdx.x * L * G::SCRATCH_PER_CTA;
    // Running weight-gradient sums [HL][2 NW][THREADS] float4, every thread its own fragments: in shared memory when
    // the host found room beside the other CTAs, else in global memory (L2).
    float4* dws = a.dw_scratch != nullptr ? reinterpret_cast<float4*>(a.dw_scratch) + (size_t)blockIdx.x * HL * 2 * NW * THREADS
                                          : reinterpret_cast<float4*>(code + a.prog.n_instr);
#ifdef QB_PHASE_TIMING
    long long phase_[10] = {0, 0, 0, 0, 0, 0, 0, 0, 0, 0};
    long long last_ = clock64();
#endif

    for (int i = tid; i < a.prog.n_instr; i += THREADS) code[i] = a.prog.code[i];
    for (int i = tid; i < L * W; i += THREADS) {
        const int l = i / W, n = i % W;
        pbias[i] = (a.b_off[l] >= 0 && n < a.width[l]) ? a.params[a.b_off[l] + n] : 0.0f;
        gbias[i] = 0.0f;
    }
    for (int i = tid; i < 4 * W; i += THREADS) {
        const int k = i / W, n = i % W;
        pfirst[i] = (k < d0 && n < a.width[0]) ? a.params[a.w_off[0] + k * a.width[0] + n] : 0.0f;
        gfirst[i] = 0.0f;
    }
    for (int i = tid; i < W; i += THREADS) {
        phead[i] = i < a.width[L - 1] ? a.params[a.w_off[L] + i] : 0.0f;
        ghead[i] = 0.0f;
    }
    if (tid < HL) wscl[tid] = a.image_scales[tid];
    if (backward)
        for (int i = tid; i < HL * 2 * NW * THREADS; i += THREADS) dws[i] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    double loss_sum = 0.0;
    float head_bias_grad = 0.0f;  // thread 0
    const float head_bias = a.b_off[L] >= 0 ? a.params[a.b_off[L]] : 0.0f;
    const float seed = a.cotangent[0] * a.weight * a.extra;
    if (tid == 0) {
        mbar_init(wbar, 1);
        mbar_init(hbar, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    __syncthreads();

    // Unit of accumulator element (j, c); its point is g for c < 2 and g + 8 above.
    auto unit_of = [&](int j, int c) { return col0 + j * 8 + 2 * t + (c & 1); };

    const int n_tiles = (int)((a.n_points + TP - 1) / TP);
    // The weight image of the next contraction is bulk-copied into shared memory as soon as the last one has been
    // read, in the order a tile uses them: forward layers 1..L-1, then L-1..1.
    const int uses_per_tile = backward ? 2 * HL : HL;
    const int my_tiles = (int)blockIdx.x < n_tiles ? (n_tiles - 1 - (int)blockIdx.x) / (int)gridDim.x + 1 : 0;
    long long loads_left = (long long)my_tiles * uses_per_tile;
    int next_use = 0;              // position of the next load in the tile's order
    uint32_t wphase = 0, hphase = 0;
    const __half* images = static_cast<const __half*>(a.weight_images);
    auto load_weights = [&]() {  // thread 0
        if (loads_left-- <= 0) return;
        const int layer = next_use < HL ? next_use : 2 * HL - 1 - next_use;
        if (++next_use == uses_per_tile) next_use = 0;
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        mbar_expect_tx(wbar, G::WIMG_BYTES);
        bulk_load(wbuf, images + (size_t)layer * 2 * WPLANE, G::WIMG_BYTES, wbar);
    };
    if (tid == 0) load_weights();

    for (int tile = blockIdx.x; tile < n_tiles; tile += gridDim.x) {
        const long long p0 = (long long)tile * TP;
        float acc[S][2][4];
        float x[2][4];
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            const long long p = min(p0 + g + 8 * i, a.n_points - 1);
#pragma unroll
            for (int k = 0; k < 4; ++k) x[i][k] = k < d0 ? a.table[p * a.ncols + k] : 0.0f;
        }

        // ------------------------------ forward ------------------------------
        for (int l = 0; l < L; ++l) {
            if (l == 0) {
#pragma unroll
                for (int s = 0; s < S; ++s)
#pragma unroll
                    for (int j = 0; j < 2; ++j)
#pragma unroll
                        for (int c = 0; c < 4; ++c) acc[s][j][c] = 0.0f;
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    if (k < d0) {
#pragma unroll
                        for (int j = 0; j < 2; ++j)
#pragma unroll
                            for (int c = 0; c < 4; ++c) {
                                const float w = pfirst[k * W + unit_of(j, c)];
                                acc[0][j][c] += x[c >> 1][k] * w;
#pragma unroll
                                for (int dj = 0; dj < SG::ndirs; ++dj) acc[SG::base(dj)][j][c] += a.dirs[dj * d0 + k] * w;
                            }
                    }
                }
            } else {
                mbar_wait(wbar, wphase, a.error);
                wphase ^= 1;
                __syncthreads();  // the previous epilogue's activations are in place
                if (backward && tid == 0) {
                    // Save layer l-1's jets for the reverse sweep: the operand planes as they sit in shared memory, one
                    // bulk copy (TMA engine).
                    asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;" ::"l"(
                                     sh + (size_t)(l - 1) * G::SCRATCH_PER_CTA),
                                 "r"(smem_u32(act)), "r"((uint32_t)G::ACT_BYTES)
                                 : "memory");
                    asm volatile("cp.async.bulk.commit_group;" ::: "memory");
                }
                QB_PHASE(0);  // wait for the weight image
                warp_contract<S, NW, LD, PLANE, WPLANE, true>(act, wbuf, scl + (l - 1) * S * NW, wscl[l - 1], warp, lane, acc);
                // The epilogue overwrites the operand: the bulk copy must have read it.
                if (backward && tid == 0) asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
                __syncthreads();
                if (tid == 0) load_weights();
                QB_PHASE(1);  // forward contraction
            }
#pragma unroll
            for (int j = 0; j < 2; ++j)
#pragma unroll
                for (int c = 0; c < 4; ++c) acc[0][j][c] += pbias[l * W + unit_of(j, c)];
            // The reverse sweep needs the pre-activation streams; of the primal one only tanh itself (z_0 for sin).
            float4* zl = reinterpret_cast<float4*>(sz + (size_t)l * G::SCRATCH_PER_CTA) + tid;
            if (backward) {
#pragma unroll
                for (int s = ACT == ACT_TANH ? 1 : 0; s < S; ++s)
#pragma unroll
                    for (int j = 0; j < 2; ++j)
                        zl[(2 * s + j) * THREADS] = make_float4(acc[s][j][0], acc[s][j][1], acc[s][j][2], acc[s][j][3]);
            }
#pragma unroll
            for (int j = 0; j < 2; ++j)
#pragma unroll
                for (int c = 0; c < 4; ++c) {
                    float v[S];
#pragma unroll
                    for (int s = 0; s < S; ++s) v[s] = acc[s][j][c];
                    jet_apply<float, SG, ACT>(v, a.merge_w);
#pragma unroll
                    for (int s = 0; s < S; ++s) acc[s][j][c] = v[s];
                }
            if (backward && ACT == ACT_TANH) {
#pragma unroll
                for (int j = 0; j < 2; ++j) zl[j * THREADS] = make_float4(acc[0][j][0], acc[0][j][1], acc[0][j][2], acc[0][j][3]);
            }
            if (l + 1 < L) {
                store_blocks<S, NW, LD, PLANE>(acc, act, scl + l * S * NW, warp, g, t);
                // The next iteration saves these planes with a bulk copy: make the writes visible to that proxy.
                if (backward) asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            }
        }

        QB_PHASE(2);  // forward epilogues (bias, saves, jets, staging of the next operand)
        // ------------------------- head and residual -------------------------
        float wh[2][2];
#pragma unroll
        for (int j = 0; j < 2; ++j)
#pragma unroll
            for (int c = 0; c < 2; ++c) wh[j][c] = phead[unit_of(j, c)];
#pragma unroll
        for (int s = 0; s < S; ++s)
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                float dot = 0.0f;
#pragma unroll
                for (int j = 0; j < 2; ++j) dot += acc[s][j][2 * i] * wh[j][0] + acc[s][j][2 * i + 1] * wh[j][1];
                dot += __shfl_xor_sync(0xffffffffu, dot, 1);
                dot += __shfl_xor_sync(0xffffffffu, dot, 2);
                if (t == 0) red[(warp * S + s) * TP + g + 8 * i] = dot;
            }
        __syncthreads();
        if (tid < TP) {
            const long long p = p0 + tid;
            const bool valid = p < a.n_points;
            const long long pc = valid ? p : a.n_points - 1;
#pragma unroll
            for (int s = 0; s < S; ++s) {
                float u = red[s * TP + tid];
#pragma unroll
                for (int q = 1; q < NW; ++q) u += red[(q * S + s) * TP + tid];
                us[s * TP + tid] = s == 0 ? u + head_bias : u;
            }
            float r[MAX_REGS];
            run_program<float>(code, a.prog.n_instr, static_cast<const float*>(a.prog.consts), a.table + pc * a.ncols,
                               us + tid, TP, r);
            if (valid) loss_sum += (double)r[a.prog.value_reg];
#pragma unroll
            for (int s = 0; s < S; ++s) {
                const int reg = a.prog.grad_regs[s];
                uh[s * TP + tid] = (valid && reg >= 0) ? seed * r[reg] : 0.0f;
            }
        }
        __syncthreads();
        QB_PHASE(3);  // head and residual program
        if (!backward) continue;

        // ------------------------------ backward ------------------------------
        auto load_jets = [&](int layer) {  // thread 0: saved jets of `layer` into ht
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            mbar_expect_tx(hbar, G::ACT_BYTES);
            bulk_load(ht, sh + (size_t)layer * G::SCRATCH_PER_CTA, G::ACT_BYTES, hbar);
        };
        if (tid == 0 && HL > 0) {
            asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");  // the saves of the forward pass are complete
            load_jets(HL - 1);
        }
        {
            // Head: dW = sum h * uhat, db = sum uhat(primal), G = uhat (x) w.
            float pw[4] = {0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll
            for (int s = 0; s < S; ++s) {
                const float u0 = uh[s * TP + g], u1 = uh[s * TP + g + 8];
#pragma unroll
                for (int j = 0; j < 2; ++j)
#pragma unroll
                    for (int c = 0; c < 4; ++c) {
                        const float u = c < 2 ? u0 : u1;
                        pw[2 * j + (c & 1)] += acc[s][j][c] * u;
                        acc[s][j][c] = u * wh[j][c & 1];
                    }
            }
            add_column_sums(pw, ghead, lane, col0, t);
            if (tid == 0) {
                float total = 0.0f;
#pragma unroll
                for (int p = 0; p < TP; ++p) total += uh[p];
                head_bias_grad += total;
            }
        }
        for (int l = L - 1; l >= 0; --l) {
            const float4* zl = reinterpret_cast<const float4*>(sz + (size_t)l * G::SCRATCH_PER_CTA) + tid;
#pragma unroll
            for (int j = 0; j < 2; ++j) {
                float z[S][4];
#pragma unroll
                for (int s = 0; s < S; ++s) {
                    const float4 q = zl[(2 * s + j) * THREADS];
                    z[s][0] = q.x; z[s][1] = q.y; z[s][2] = q.z; z[s][3] = q.w;
                }
#pragma unroll
                for (int c = 0; c < 4; ++c) {
                    float zc[S], gc[S];
#pragma unroll
                    for (int s = 0; s < S; ++s) {
                        zc[s] = z[s][c];
                        gc[s] = acc[s][j][c];
                    }
                    if (ACT == ACT_TANH)
                        jet_apply_transposed_with<float, SG>(TanhD<float>(zc[0]), zc, gc, a.merge_w);
                    else
                        jet_apply_transposed<float, SG, ACT>(zc, gc, a.merge_w);
#pragma unroll
                    for (int s = 0; s < S; ++s) acc[s][j][c] = gc[s];
                }
            }
            {
                float pb[4];
#pragma unroll
                for (int j = 0; j < 2; ++j) {
                    pb[2 * j] = acc[0][j][0] + acc[0][j][2];
                    pb[2 * j + 1] = acc[0][j][1] + acc[0][j][3];
                }
                add_column_sums(pb, gbias + l * W, lane, col0, t);
            }
            if (l == 0) {
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    if (k < d0) {
                        float pw[4] = {0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll
                        for (int j = 0; j < 2; ++j)
#pragma unroll
                            for (int c = 0; c < 4; ++c) {
                                float v = x[c >> 1][k] * acc[0][j][c];
#pragma unroll
                                for (int dj = 0; dj < SG::ndirs; ++dj) v += a.dirs[dj * d0 + k] * acc[SG::base(dj)][j][c];
                                pw[2 * j + (c & 1)] += v;
                            }
                        add_column_sums(pw, gfirst + k * W, lane, col0, t);
                    }
                }
                break;
            }
            QB_PHASE(4);  // transposed jets, bias partials
            // Cotangents of the pre-activations: operand of both contractions below.
            store_blocks<S, NW, LD, PLANE>(acc, act, scl_z, warp, g, t);
            mbar_wait(hbar, hphase, a.error);
            hphase ^= 1;
            __syncthreads();
            QB_PHASE(5);  // backward staging
            // Weight gradient: dW[k][n] += sum_rows H[row][k] * Zhat[row][n]; this warp: its 16 k x all n.
            {
                float4* gw = dws + (size_t)(l - 1) * 2 * NW * THREADS + tid;
                // Starts from the running sums, loaded before the loop so that their latency hides behind the contraction.
                float dw[NW][2][4];
#pragma unroll
                for (int nb = 0; nb < NW; ++nb)
#pragma unroll
                    for (int j = 0; j < 2; ++j) {
                        const float4 q = gw[(2 * nb + j) * THREADS];
                        dw[nb][j][0] = q.x; dw[nb][j][1] = q.y; dw[nb][j][2] = q.z; dw[nb][j][3] = q.w;
                    }
                const int mi = lane >> 3, rr = lane & 7;
                const __half* a_lane = ht + ((mi >> 1) * 8 + rr) * LD + col0 + (mi & 1) * 8;
                const __half* b_lane = act + ((mi & 1) * 8 + rr) * LD + (mi >> 1) * 8;
                const float* scl_h = scl + (l - 1) * S * NW;
#pragma unroll
                for (int s = 0; s < S; ++s) {
                    uint32_t ahi[4], alo[4];
                    ldmatrix_x4<true>(ahi, a_lane + s * 16 * LD);
                    ldmatrix_x4<true>(alo, a_lane + s * 16 * LD + PLANE);
                    const float fh = scl_h[s * NW + warp];
#pragma unroll
                    for (int nb = 0; nb < NW; ++nb) {
                        uint32_t bhi[4], blo[4];
                        ldmatrix_x4<true>(bhi, b_lane + s * 16 * LD + nb * 16);
                        ldmatrix_x4<true>(blo, b_lane + s * 16 * LD + nb * 16 + PLANE);
                        mma_step(dw[nb], ahi, alo, bhi, blo, fh * scl_z[s * NW + nb]);
                    }
                }
#pragma unroll
                for (int nb = 0; nb < NW; ++nb)
#pragma unroll
                    for (int j = 0; j < 2; ++j)
                        gw[(2 * nb + j) * THREADS] = make_float4(dw[nb][j][0], dw[nb][j][1], dw[nb][j][2], dw[nb][j][3]);
            }
            QB_PHASE(6);  // weight gradient
            // Cotangents of layer l-1's jets: G = Zhat W^T.
            mbar_wait(wbar, wphase, a.error);
            wphase ^= 1;
            warp_contract<S, NW, LD, PLANE, WPLANE, false>(act, wbuf, scl_z, wscl[l - 1], warp, lane, acc);
            __syncthreads();
            if (tid == 0) {
                load_weights();
                if (l > 1) load_jets(l - 2);
            }
            QB_PHASE(7);  // data gradient
        }
    }
#ifdef QB_PHASE_TIMING
    if (tid == 0 && blockIdx.x == 0) {
        printf("phases S=%d W=%d tiles=%d:", S, W, my_tiles);
        for (int i = 0; i < 8; ++i) printf(" %lld", phase_[i] / max(my_tiles, 1));
        printf("\n");
    }
#endif

    // Per-CTA gradients in parameter order, and the loss partial, in a fixed order.
    __syncthreads();
    if (backward) {
        float* my_grad = a.grad_cta + (size_t)blockIdx.x * a.P;
        for (int i = tid; i < L * W; i += THREADS) {
            const int l = i / W, n = i % W;
            if (a.b_off[l] >= 0 && n < a.width[l]) my_grad[a.b_off[l] + n] = gbias[i];
        }
        for (int i = tid; i < d0 * W; i += THREADS) {
            const int k = i / W, n = i % W;
            if (n < a.width[0]) my_grad[a.w_off[0] + k * a.width[0] + n] = gfirst[i];
        }
        for (int i = tid; i < a.width[L - 1]; i += THREADS) my_grad[a.w_off[L] + i] = ghead[i];
        if (tid == 0 && a.b_off[L] >= 0) my_grad[a.b_off[L]] = head_bias_grad;
        for (int l = 1; l < L; ++l) {
            const int rows = a.width[l - 1], cols = a.width[l];
            float* out = my_grad + a.w_off[l];
            for (int q = 0; q < 2 * NW; ++q) {
                float4 v = dws[((size_t)(l - 1) * 2 * NW + q) * THREADS + tid];
                v.x = fmaf(v.x, MMA_TRUNCATION, v.x);
                v.y = fmaf(v.y, MMA_TRUNCATION, v.y);
                v.z = fmaf(v.z, MMA_TRUNCATION, v.z);
                v.w = fmaf(v.w, MMA_TRUNCATION, v.w);
                const int k = col0 + g, n = (q >> 1) * 16 + (q & 1) * 8 + 2 * t;
                if (k < rows && n < cols) out[k * cols + n] = v.x;
                if (k < rows && n + 1 < cols) out[k * cols + n + 1] = v.y;
                if (k + 8 < rows && n < cols) out[(k + 8) * cols + n] = v.z;
                if (k + 8 < rows && n + 1 < cols) out[(k + 8) * cols + n + 1] = v.w;
            }
        }
    }
    double* lred = reinterpret_cast<double*>(red);
    static_assert(4 * NW * G::ROWS >= 8 * TP || S == 1, "loss partials fit the reduction area");
    double* lsum = S == 1 ? reinterpret_cast<double*>(act) : lred;
    if (tid < TP) lsum[tid] = loss_sum;
    __syncthreads();
    if (tid == 0) {
        double total = 0.0;
        for (int p = 0; p < TP; ++p) total += lsum[p];
        a.loss_cta[blockIdx.x] = total;
    }
}

}  // namespace qb
