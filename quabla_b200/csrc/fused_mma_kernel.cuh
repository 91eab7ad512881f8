// Fused engine, float32, hidden widths up to 64, weight contractions on the tensor cores with operands split into
// three bfloat16 parts.
//
// Split.  x = hi + mid + lo with hi = bf16(x), mid = bf16(x - hi) and lo the rest, which is a bfloat16 as well: 24 bits in
// three parts of 8, every element with an exponent of its own and float32's range, so the split loses nothing.  A
// product A.B is hi.hi + (hi.mid + mid.hi) + (mid.mid + hi.lo + lo.hi); the dropped mid.lo, lo.mid and lo.lo are below
// 2^-25 of it and of random sign.  The tensor core truncates what it adds, a loss of one sign that no number of points
// averages out, so hi.hi runs twice, the second time onto minus its own result: that leaves exactly what the first run
// dropped, and the smaller products are added to it.  Seven m16n8k16 instructions per 16 contraction elements.  Mean
// relative loss of such a step, <error, exact> / <exact, exact> over 500,000 sums of 16 products against float64: 6e-12
// (normal operands), 1.3e-11 (uniform), 1.2e-9 (positive), 1.5e-10 (exponents spread by 2^40); of hi.hi run once 0.8e-8 to
// 3.7e-8, a factor that changes with the operands and cannot be put back by a constant.
//
// Same structure as fused_step_kernel (fused_kernel.cuh): persistent CTAs walk tiles of 16 points, run forward /
// residual / reverse sweep per tile, keep the saved jets in an L2-resident per-CTA scratch and accumulate weight
// gradients per CTA.  Warp w owns units 16 w .. 16 w + 15 (W / 16 warps): for every stream the 16 x 16 tile
// (points x units) as two m16n8 accumulator fragments, so thread (g = lane / 4, t = lane % 4) holds points
// {g, g + 8} x units {2t, 2t + 1} of both fragments for ALL streams, and the jet composition stays register-only.
// Networks narrower than W (or of unequal widths) run padded with zero weights: a padded unit's activation meets
// only zero weights and its cotangent is zero.
//
// Bound: the contractions, 63 % of a tile's cycles (width 64, four streams: 69,000 cycles per tile with two CTAs on an SM;
// head and residual program 10 %, transposed jets 8 %, staging 3 %), in which the tensor pipe is busy 70 % of the time (45 %
// over all), and the number of CTAs that overlap one another's other phases: shared memory holds two of 80 KB.
// Measured, microseconds per step or call at width 64 (50) with three tf32 products or, at width 50, layer by layer; with two
// float16 parts; and now: 65,536-point 2-D Poisson 727, 407, 597; 10,007-point gradients 595, 204, 240; 1,048,576-point beam
// 11,150, 7,250, 9,990; 20,000 points at width 50 848, 155, 218.  Error of float32 gradients against float64 in
// parts of the first of these (geometric mean over four workloads, two activations, two weight scales, six seeds, 1,003 and 20,011
// points): 0.65, 0.59, 0.69, 0.59 and 0.64 at widths 16, 24, 32, 48 and 50, where the former kernels multiplied and added in
// float32, and 0.08 at width 64.  Two float16 parts with an exponent per 16 x 16 block were 1.15 to 1.33 times as far off and lost
// entries that are small beside their neighbours altogether (5e-2 of themselves at 2^-30).
//
// Replaces the reference's per-node plan execution (crates/quabla-core/src/tensor_ir/cuda.rs:1792-2972) and its
// cuBLAS strided-batched GEMV-shaped calls (cuda.rs:4936-5035).
#pragma once
#include <cuda_bf16.h>

#include <cstdint>
#include <cstdio>

#include "fused.h"
#include "fused_kernel.cuh"

namespace qb {

// Four 8x8 matrices of 16-bit elements; thread (g, t) receives elements 2t, 2t + 1 of row g of each (TRANS: of
// column g), the m16n8k16 fragment layouts.
template <bool TRANS>
__device__ __forceinline__ void ldmatrix_x4(uint32_t (&r)[4], const __nv_bfloat16* row_ptr) {
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

// d += a (16x16, row) * b (16x8, col), bfloat16 operands, float32 accumulate.  Not volatile: the accumulator operands
// carry the dependencies, the compiler may interleave independent chains.
__device__ __forceinline__ void mma_bf16(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

// N steps of 16 x 16 by 16 x 16 on {hi, mid, lo} fragments, of A(n) and B(n) each: acc[n] += (hi.hi as the tensor
// core leaves it) + (what it left out and the five smaller products).  The 2 N chains of seven dependent instructions
// are issued side by side (one pair of streams at a time instead of one: 1 to 3 % of a step).
template <int N, typename FragA, typename FragB>
__device__ __forceinline__ void mma_steps(float (*acc)[2][4], FragA A, FragB B) {
    constexpr int PRODUCTS[7][2] = {{0, 0}, {0, 0}, {2, 0}, {0, 2}, {1, 1}, {1, 0}, {0, 1}};
    float part[N][2][4], rest[N][2][4];
#pragma unroll
    for (int q = 0; q < 7; ++q)
#pragma unroll
        for (int n = 0; n < N; ++n)
#pragma unroll
            for (int j = 0; j < 2; ++j) {
                float(&d)[4] = rest[n][j];
                if (q == 0) d[0] = d[1] = d[2] = d[3] = 0.0f;
                const uint32_t(&b)[4] = B(n)[PRODUCTS[q][1]];
                mma_bf16(d, A(n)[PRODUCTS[q][0]], b[2 * j], b[2 * j + 1]);
#pragma unroll
                for (int c = 0; c < 4; ++c) {
                    if (q == 0) {
                        part[n][j][c] = d[c];
                        d[c] = -d[c];
                    }
                    if (q == 6) acc[n][j][c] += part[n][j][c] + d[c];
                }
            }
}

// Two elements as packed bfloat16 {hi, mid, lo} pairs.
__device__ __forceinline__ void split_bf16(float x0, float x1, uint32_t (&parts)[3]) {
#pragma unroll
    for (int q = 0; q < 3; ++q) {
        const __nv_bfloat162 pair = __floats2bfloat162_rn(x0, x1);
        parts[q] = *reinterpret_cast<const uint32_t*>(&pair);
        x0 -= __uint_as_float(parts[q] << 16);
        x1 -= __uint_as_float(parts[q] & 0xffff0000u);
    }
}

// Operand planes: rows of W elements in chunks of eight, laid out so that the eight row addresses of an ldmatrix tile
// (one chunk of eight successive rows) fall into distinct bank groups: padded by a chunk, or, at width 64, where the
// padding would cost a resident CTA at six streams, unpadded with the chunks of a row permuted by its number.
template <int W>
struct PlaneLayout {
    static constexpr int LD = W == 64 ? 64 : W + 8;
    static __host__ __device__ constexpr int at(int row, int chunk) { return row * LD + 8 * (W == 64 ? chunk ^ (row & 7) : chunk); }
};

// ---- asynchronous staging: bulk copies (TMA engine, no multicast) ----
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

// Weight images written by prep_weights_kernel, one per hidden-to-hidden layer: {hi, mid, lo} planes [W][W] of the
// row-major [in][out] matrix, zero-padded to W x W.  The forward contraction reads it transposed (ldmatrix .trans), the
// data gradient as it is.
struct PrepArgs {
    int layers;                       // hidden-to-hidden layers
    int w_off[FUSED_MAX_LAYERS + 1];  // parameter offset of network layer 1 + i
    int rows[FUSED_MAX_LAYERS + 1];   // its true input and output widths
    int cols[FUSED_MAX_LAYERS + 1];
};

template <int W>
static __global__ void __launch_bounds__(256) prep_weights_kernel(const float* __restrict__ params, PrepArgs p,
                                                                  uint32_t* __restrict__ images) {
    typedef PlaneLayout<W> P;
    const int layer = blockIdx.y, rows = p.rows[layer], cols = p.cols[layer];
    const float* w = params + p.w_off[layer];
    constexpr int PLANE = W * P::LD / 2;  // 32-bit words
    uint32_t* img = images + (size_t)layer * 3 * PLANE;
    for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < W * W / 2; e += gridDim.x * blockDim.x) {
        const int r = e / (W / 2), c = 2 * (e % (W / 2));
        uint32_t parts[3];
        split_bf16((r < rows && c < cols) ? w[r * cols + c] : 0.0f, (r < rows && c + 1 < cols) ? w[r * cols + c + 1] : 0.0f, parts);
#pragma unroll
        for (int q = 0; q < 3; ++q) img[q * PLANE + (P::at(r, c / 8) + c % 8) / 2] = parts[q];
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
    static constexpr int LD = PlaneLayout<W>::LD;
    static constexpr int PLANE = ROWS * LD;      // elements per operand plane
    static constexpr int WPLANE = W * LD;        // elements per weight plane
    static constexpr int ACT_BYTES = 6 * PLANE;  // hi, mid and lo
    static constexpr int WIMG_BYTES = 6 * WPLANE;
    static constexpr int OFF_ACT = 0;                      // activations / cotangents, [hi, mid, lo][ROWS][LD]
    static constexpr int OFF_HT = OFF_ACT + ACT_BYTES;     // previous layer's jets (weight-gradient operand), same layout
    static constexpr int OFF_WB = OFF_HT + ACT_BYTES;      // weight image of the contraction at hand
    static constexpr int OFF_RED = OFF_WB + WIMG_BYTES;    // [NW][S][TP] output-layer partials
    static constexpr int OFF_U = OFF_RED + 4 * NW * ROWS;  // [S][TP]
    static constexpr int OFF_UH = OFF_U + 4 * ROWS;        // [S][TP]
    static constexpr int OFF_BAR = OFF_UH + 4 * ROWS;      // two mbarriers
    static constexpr int OFF_VAR = OFF_BAR + 16;           // regions that depend on the depth:
    // parameters {biases [L][W], first layer [4][W], output layer [W]} and gradient sums of the same
    static __host__ __device__ constexpr size_t base_bytes(int L) { return (size_t)OFF_VAR + 4 * 2 * (size_t)(L + 5) * W; }
    static constexpr size_t DW_BYTES = 4 * (size_t)W * W;  // running weight-gradient sums of one layer
    // CTAs that share an SM: as many as its shared memory holds of a network of four hidden layers, and up to 12 warps of
    // 168 registers a thread (up to four streams) or 8 of 224 to 255.
    static constexpr int FIT = (int)(FUSED_SM_SMEM / (base_bytes(4) + FUSED_CTA_SMEM + 512));
    static constexpr int BY_REGISTERS = (S <= 4 ? 12 : 8) / NW;
    static constexpr int MIN_CTAS = FIT < 1 ? 1 : FIT < BY_REGISTERS ? FIT : BY_REGISTERS;
    // Saved jets: the operand planes as they sit in shared memory, one bulk copy per layer.  Saved pre-activations:
    // read back by the thread that wrote them, so laid out per thread.
    static constexpr size_t SCRATCH_PER_CTA = (size_t)ACT_BYTES / 4;
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

// The warp's 16 x 16 block of every stream, split, into the operand planes.
template <int S, int W>
__device__ __forceinline__ void store_blocks(const float (&acc)[S][2][4], __nv_bfloat16* planes, int warp, int g, int t) {
    typedef PlaneLayout<W> P;
    constexpr int PLANE = S * 16 * P::LD / 2;  // 32-bit words
    uint32_t* words = reinterpret_cast<uint32_t*>(planes);
#pragma unroll
    for (int s = 0; s < S; ++s)
#pragma unroll
        for (int j = 0; j < 2; ++j)
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                uint32_t parts[3];
                split_bf16(acc[s][j][2 * i], acc[s][j][2 * i + 1], parts);
#pragma unroll
                for (int q = 0; q < 3; ++q) words[q * PLANE + P::at(s * 16 + 8 * i + g, 2 * warp + j) / 2 + t] = parts[q];
            }
}

// acc[s] = A[rows of stream s][W] * B[W][16 columns of this warp].  FORWARD: B(k, n) = W[k][n]; else B(k, n) = W[n][k].
template <int S, int W, bool FORWARD>
__device__ __forceinline__ void warp_contract(const __nv_bfloat16* __restrict__ A, const __nv_bfloat16* __restrict__ Wimg,
                                              int warp, int lane, float (&acc)[S][2][4]) {
    typedef PlaneLayout<W> P;
    constexpr int PLANE = S * 16 * P::LD, WPLANE = W * P::LD;
#pragma unroll
    for (int s = 0; s < S; ++s)
#pragma unroll
        for (int j = 0; j < 2; ++j)
#pragma unroll
            for (int c = 0; c < 4; ++c) acc[s][j][c] = 0.0f;
    const int mi = lane >> 3, rr = lane & 7, low = mi & 1, high = mi >> 1;
#pragma unroll
    for (int kb = 0; kb < W / 16; ++kb) {
        uint32_t b[3][4];
        const int b_at = FORWARD ? P::at(16 * kb + 8 * low + rr, 2 * warp + high) : P::at(16 * warp + 8 * high + rr, 2 * kb + low);
#pragma unroll
        for (int q = 0; q < 3; ++q) ldmatrix_x4<FORWARD>(b[q], Wimg + q * WPLANE + b_at);
        uint32_t a[2][3][4];
        auto load_a = [&](int s) {
#pragma unroll
            for (int q = 0; q < 3; ++q) ldmatrix_x4<false>(a[s & 1][q], A + q * PLANE + P::at(16 * s + 8 * low + rr, 2 * kb + high));
        };
        auto frag_b = [&](int) -> const uint32_t(&)[3][4] { return b; };
#pragma unroll
        for (int s = 0; s + 1 < S; s += 2) {
            load_a(s);
            load_a(s + 1);
            mma_steps<2>(acc + s, [&](int n) -> const uint32_t(&)[3][4] { return a[n]; }, frag_b);
        }
        if (S % 2 == 1) {
            load_a(S - 1);
            mma_steps<1>(acc + S - 1, [&](int) -> const uint32_t(&)[3][4] { return a[(S - 1) & 1]; }, frag_b);
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
    constexpr int THREADS = G::THREADS, NW = G::NW, S = G::S, TP = G::TP, PLANE = G::PLANE, WPLANE = G::WPLANE;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __nv_bfloat16* act = reinterpret_cast<__nv_bfloat16*>(smem_raw + G::OFF_ACT);
    __nv_bfloat16* ht = reinterpret_cast<__nv_bfloat16*>(smem_raw + G::OFF_HT);
    __nv_bfloat16* wbuf = reinterpret_cast<__nv_bfloat16*>(smem_raw + G::OFF_WB);
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
    float* pbias = reinterpret_cast<float*>(smem_raw + G::OFF_VAR);  // [L][W]
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
    const __nv_bfloat16* images = static_cast<const __nv_bfloat16*>(a.weight_images);
    auto load_weights = [&]() {  // thread 0
        if (loads_left-- <= 0) return;
        const int layer = next_use < HL ? next_use : 2 * HL - 1 - next_use;
        if (++next_use == uses_per_tile) next_use = 0;
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        mbar_expect_tx(wbar, G::WIMG_BYTES);
        bulk_load(wbuf, images + (size_t)layer * 3 * WPLANE, G::WIMG_BYTES, wbar);
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
                warp_contract<S, W, true>(act, wbuf, warp, lane, acc);
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
                store_blocks<S, W>(acc, act, warp, g, t);
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
            store_blocks<S, W>(acc, act, warp, g, t);
            mbar_wait(hbar, hphase, a.error);
            hphase ^= 1;
            __syncthreads();
            QB_PHASE(5);  // backward staging
            // Weight gradient: dW[k][n] += sum_rows H[row][k] * Zhat[row][n]; this warp: its 16 k x all n.
            {
                float4* gw = dws + (size_t)(l - 1) * 2 * NW * THREADS + tid;
                // The running sums, loaded before the loop so that their latency hides behind the contraction, take this tile's
                // in one addition.
                float4 sums[NW][2];
                float dw[NW][2][4];
#pragma unroll
                for (int nb = 0; nb < NW; ++nb)
#pragma unroll
                    for (int j = 0; j < 2; ++j) {
                        sums[nb][j] = gw[(2 * nb + j) * THREADS];
#pragma unroll
                        for (int c = 0; c < 4; ++c) dw[nb][j][c] = 0.0f;
                    }
                typedef PlaneLayout<W> P;
                const int mi = lane >> 3, rr = lane & 7, low = mi & 1, high = mi >> 1;
#pragma unroll
                for (int s = 0; s < S; ++s) {
                    uint32_t ha[3][4];
#pragma unroll
                    for (int q = 0; q < 3; ++q) ldmatrix_x4<true>(ha[q], ht + q * PLANE + P::at(16 * s + 8 * high + rr, 2 * warp + low));
                    uint32_t zb[2][3][4];
                    auto load_b = [&](int nb) {
#pragma unroll
                        for (int q = 0; q < 3; ++q)
                            ldmatrix_x4<true>(zb[nb & 1][q], act + q * PLANE + P::at(16 * s + 8 * low + rr, 2 * nb + high));
                    };
                    auto frag_a = [&](int) -> const uint32_t(&)[3][4] { return ha; };
#pragma unroll
                    for (int nb = 0; nb + 1 < NW; nb += 2) {
                        load_b(nb);
                        load_b(nb + 1);
                        mma_steps<2>(dw + nb, frag_a, [&](int n) -> const uint32_t(&)[3][4] { return zb[n]; });
                    }
                    if (NW % 2 == 1) {
                        load_b(NW - 1);
                        mma_steps<1>(dw + NW - 1, frag_a,
                                     [&](int) -> const uint32_t(&)[3][4] { return zb[(NW - 1) & 1]; });
                    }
                }
#pragma unroll
                for (int nb = 0; nb < NW; ++nb)
#pragma unroll
                    for (int j = 0; j < 2; ++j) {
                        const float4 q = sums[nb][j];
                        gw[(2 * nb + j) * THREADS] =
                            make_float4(q.x + dw[nb][j][0], q.y + dw[nb][j][1], q.z + dw[nb][j][2], q.w + dw[nb][j][3]);
                    }
            }
            QB_PHASE(6);  // weight gradient
            // Cotangents of layer l-1's jets: G = Zhat W^T.
            mbar_wait(wbar, wphase, a.error);
            wphase ^= 1;
            warp_contract<S, W, false>(act, wbuf, warp, lane, acc);
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
                const float4 v = dws[((size_t)(l - 1) * 2 * NW + q) * THREADS + tid];
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
