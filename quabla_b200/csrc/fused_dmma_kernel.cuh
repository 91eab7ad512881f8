// Fused engine, float64, hidden widths up to 64, weight contractions on the FP64 tensor-core path (mma.sync m8n8k4).
//
// The float64 sibling of fused_mma_kernel (same phases, same per-CTA gradient sums, same padding): tiles of 8 points,
// warp w owns units 16 w .. 16 w + 15, and thread (g = lane / 4, t = lane % 4) holds point g x units {2t, 2t + 1} of two
// 8-unit blocks for ALL streams.  FP64 MMA and FP64 FMA share one pipe of 64 multiply-adds per cycle and SM, so the
// kernel is bound by that pipe once a few warps per scheduler hide its latency: the operands go through shared
// memory as plain doubles (rows of W + 4: a half warp's 64-bit fragment reads fall into 16 distinct bank pairs in
// all four access patterns), weights as padded images loaded by one bulk copy per use.  Tiles of 8 points rather
// than 16 halve a thread's sums and the tile's shared memory, and give small point sets twice the CTAs.
#pragma once
#include "dmma_gemm.cuh"  // dmma_m8n8k4
#include "fused_mma_kernel.cuh"  // bulk copies, barriers

namespace qb {

// Weight images: the row-major [in][out] matrices zero-padded to [W][W + 4], one per hidden-to-hidden layer.
static __global__ void __launch_bounds__(256) prep_weights64_kernel(const double* __restrict__ params, PrepArgs p, int W,
                                                                    double* __restrict__ images) {
    const int layer = blockIdx.y, rows = p.rows[layer], cols = p.cols[layer], ld = W + 4;
    const double* w = params + p.w_off[layer];
    double* img = images + (size_t)layer * W * ld;
    for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < W * ld; e += gridDim.x * blockDim.x) {
        const int r = e / ld, c = e % ld;
        img[e] = (r < rows && c < cols) ? w[r * cols + c] : 0.0;
    }
}

template <int CODE, int W_>
struct DmmaGeom {
    typedef Sig<CODE> sig;
    static constexpr int W = W_;
    static constexpr int S = sig::S;
    static constexpr int NW = W / 16;
    static constexpr int THREADS = 32 * NW;
    static constexpr int TP = 8;
    static constexpr int ROWS = S * TP;
    static constexpr int LD = W + 4;
    static constexpr int ACT_BYTES = 8 * ROWS * LD;
    static constexpr int WIMG_BYTES = 8 * W * LD;
    static constexpr int OFF_ACT = 0;
    static constexpr int OFF_HT = OFF_ACT + ACT_BYTES;
    static constexpr int OFF_WB = OFF_HT + ACT_BYTES;
    static constexpr int OFF_RED = OFF_WB + WIMG_BYTES;    // [NW][S][TP] output-layer partials
    static constexpr int OFF_U = OFF_RED + 8 * NW * ROWS;  // [S][TP]
    static constexpr int OFF_UH = OFF_U + 8 * ROWS;        // [S][TP]
    static constexpr int OFF_BAR = OFF_UH + 8 * ROWS;      // two mbarriers
    static constexpr int OFF_VAR = OFF_BAR + 16;
    // parameters {biases [L][W], first layer [4][W], output layer [W]} and gradient sums of the same
    static __host__ __device__ constexpr size_t base_bytes(int L) { return (size_t)OFF_VAR + 8 * 2 * (size_t)(L + 5) * W; }
    static constexpr size_t DW_BYTES = 8 * (size_t)W * W;
    static constexpr int MIN_CTAS = (S <= 4 ? 12 : 8) / NW;
    static constexpr size_t SCRATCH_PER_CTA = (size_t)ROWS * LD;
};

// acc[s] = A[rows of stream s][W] * B[W][16 columns of this warp].  FORWARD: B(k, n) = W[k][n]; else B(k, n) = W[n][k].
template <int S, int W, int LD, bool FORWARD>
__device__ __forceinline__ void warp_contract64(const double* __restrict__ A, const double* __restrict__ Wimg, int warp, int g,
                                                int t, double (&acc)[S][2][2]) {
#pragma unroll
    for (int s = 0; s < S; ++s)
#pragma unroll
        for (int j = 0; j < 2; ++j) acc[s][j][0] = acc[s][j][1] = 0.0;
    const double* a_lane = A + g * LD + t;
    const double* b_lane = FORWARD ? Wimg + t * LD + 16 * warp + g : Wimg + (16 * warp + g) * LD + t;
#pragma unroll 4
    for (int k = 0; k < W; k += 4) {
        const double b0 = b_lane[FORWARD ? k * LD : k], b1 = b_lane[FORWARD ? k * LD + 8 : k + 8 * LD];
#pragma unroll
        for (int s = 0; s < S; ++s) {
            const double av = a_lane[s * 8 * LD + k];
            dmma_m8n8k4(acc[s][0], av, b0);
            dmma_m8n8k4(acc[s][1], av, b1);
        }
    }
}

// Column sums over the 8 points of the warp's block; lanes with g == 0 add them to dst, which only this warp touches.
__device__ __forceinline__ void add_column_sums64(double (&v)[4], double* dst, int lane, int col0, int t) {
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
__global__ void __launch_bounds__(DmmaGeom<CODE, W>::THREADS, DmmaGeom<CODE, W>::MIN_CTAS) fused_dmma_kernel(FusedArgs<double> a) {
    typedef DmmaGeom<CODE, W> G;
    typedef Sig<CODE> SG;
    constexpr int THREADS = G::THREADS, NW = G::NW, S = G::S, TP = G::TP, LD = G::LD;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    double* act = reinterpret_cast<double*>(smem_raw + G::OFF_ACT);
    double* ht = reinterpret_cast<double*>(smem_raw + G::OFF_HT);
    double* wbuf = reinterpret_cast<double*>(smem_raw + G::OFF_WB);
    double* red = reinterpret_cast<double*>(smem_raw + G::OFF_RED);
    double* us = reinterpret_cast<double*>(smem_raw + G::OFF_U);
    double* uh = reinterpret_cast<double*>(smem_raw + G::OFF_UH);
    uint64_t* wbar = reinterpret_cast<uint64_t*>(smem_raw + G::OFF_BAR);
    uint64_t* hbar = wbar + 1;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int g = lane >> 2, t = lane & 3;
    const int col0 = warp * 16;
    const int L = a.L, d0 = a.d0, HL = L - 1;
    const bool backward = a.forward_only == 0;
    double* pbias = reinterpret_cast<double*>(smem_raw + G::OFF_VAR);
    double* pfirst = pbias + L * W;
    double* phead = pfirst + 4 * W;
    double* gbias = phead + W;
    double* gfirst = gbias + L * W;
    double* ghead = gfirst + 4 * W;
    int4* code = reinterpret_cast<int4*>(smem_raw + G::base_bytes(L));
    double* sz = a.scratch_z + (size_t)blockIdx.x * L * G::SCRATCH_PER_CTA;
    double* sh = a.scratch_h + (size_t)blockIdx.x * L * G::SCRATCH_PER_CTA;
    // Running weight-gradient sums [HL][4 NW][THREADS] double2, every thread its own fragments.
    double2* dws = a.dw_scratch != nullptr ? reinterpret_cast<double2*>(a.dw_scratch) + (size_t)blockIdx.x * HL * 4 * NW * THREADS
                                           : reinterpret_cast<double2*>(code + a.prog.n_instr);

    for (int i = tid; i < a.prog.n_instr; i += THREADS) code[i] = a.prog.code[i];
    for (int i = tid; i < L * W; i += THREADS) {
        const int l = i / W, n = i % W;
        pbias[i] = (a.b_off[l] >= 0 && n < a.width[l]) ? a.params[a.b_off[l] + n] : 0.0;
        gbias[i] = 0.0;
    }
    for (int i = tid; i < 4 * W; i += THREADS) {
        const int k = i / W, n = i % W;
        pfirst[i] = (k < d0 && n < a.width[0]) ? a.params[a.w_off[0] + k * a.width[0] + n] : 0.0;
        gfirst[i] = 0.0;
    }
    for (int i = tid; i < W; i += THREADS) {
        phead[i] = i < a.width[L - 1] ? a.params[a.w_off[L] + i] : 0.0;
        ghead[i] = 0.0;
    }
    if (backward)
        for (int i = tid; i < HL * 4 * NW * THREADS; i += THREADS) dws[i] = make_double2(0.0, 0.0);
    double loss_sum = 0.0;
    double head_bias_grad = 0.0;  // thread 0
    const double head_bias = a.b_off[L] >= 0 ? a.params[a.b_off[L]] : 0.0;
    const double seed = a.cotangent[0] * a.weight * a.extra;
    if (tid == 0) {
        mbar_init(wbar, 1);
        mbar_init(hbar, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    __syncthreads();

    // Unit of accumulator element (j, c); its point is g.
    auto unit_of = [&](int j, int c) { return col0 + j * 8 + 2 * t + c; };

    const int n_tiles = (int)((a.n_points + TP - 1) / TP);
    // Weight images in the order a tile uses them: forward layers 1..L-1, then L-1..1 (see fused_mma_kernel).
    const int uses_per_tile = backward ? 2 * HL : HL;
    const int my_tiles = (int)blockIdx.x < n_tiles ? (n_tiles - 1 - (int)blockIdx.x) / (int)gridDim.x + 1 : 0;
    long long loads_left = (long long)my_tiles * uses_per_tile;
    int next_use = 0;
    uint32_t wphase = 0, hphase = 0;
    const double* images = static_cast<const double*>(a.weight_images);
    auto load_weights = [&]() {  // thread 0
        if (loads_left-- <= 0) return;
        const int layer = next_use < HL ? next_use : 2 * HL - 1 - next_use;
        if (++next_use == uses_per_tile) next_use = 0;
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        mbar_expect_tx(wbar, G::WIMG_BYTES);
        bulk_load(wbuf, images + (size_t)layer * W * LD, G::WIMG_BYTES, wbar);
    };
    if (tid == 0) load_weights();

    for (int tile = blockIdx.x; tile < n_tiles; tile += gridDim.x) {
        const long long p0 = (long long)tile * TP;
        double acc[S][2][2];
        double x[4];
        {
            const long long p = min(p0 + g, a.n_points - 1);
#pragma unroll
            for (int k = 0; k < 4; ++k) x[k] = k < d0 ? a.table[p * a.ncols + k] : 0.0;
        }

        // ------------------------------ forward ------------------------------
        for (int l = 0; l < L; ++l) {
            if (l == 0) {
#pragma unroll
                for (int s = 0; s < S; ++s)
#pragma unroll
                    for (int j = 0; j < 2; ++j) acc[s][j][0] = acc[s][j][1] = 0.0;
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    if (k < d0) {
#pragma unroll
                        for (int j = 0; j < 2; ++j)
#pragma unroll
                            for (int c = 0; c < 2; ++c) {
                                const double w = pfirst[k * W + unit_of(j, c)];
                                acc[0][j][c] += x[k] * w;
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
                    asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;" ::"l"(
                                     sh + (size_t)(l - 1) * G::SCRATCH_PER_CTA),
                                 "r"(smem_u32(act)), "r"((uint32_t)G::ACT_BYTES)
                                 : "memory");
                    asm volatile("cp.async.bulk.commit_group;" ::: "memory");
                }
                warp_contract64<S, W, LD, true>(act, wbuf, warp, g, t, acc);
                if (backward && tid == 0) asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
                __syncthreads();
                if (tid == 0) load_weights();
            }
#pragma unroll
            for (int j = 0; j < 2; ++j)
#pragma unroll
                for (int c = 0; c < 2; ++c) acc[0][j][c] += pbias[l * W + unit_of(j, c)];
            // The reverse sweep needs the pre-activation streams; of the primal one only tanh itself (z_0 for sin).
            double2* zl = reinterpret_cast<double2*>(sz + (size_t)l * G::SCRATCH_PER_CTA) + tid;
            if (backward) {
#pragma unroll
                for (int s = ACT == ACT_TANH ? 1 : 0; s < S; ++s)
#pragma unroll
                    for (int j = 0; j < 2; ++j) zl[(2 * s + j) * THREADS] = make_double2(acc[s][j][0], acc[s][j][1]);
            }
#pragma unroll
            for (int j = 0; j < 2; ++j)
#pragma unroll
                for (int c = 0; c < 2; ++c) {
                    double v[S];
#pragma unroll
                    for (int s = 0; s < S; ++s) v[s] = acc[s][j][c];
                    jet_apply<double, SG, ACT>(v, a.merge_w);
#pragma unroll
                    for (int s = 0; s < S; ++s) acc[s][j][c] = v[s];
                }
            if (backward && ACT == ACT_TANH) {
#pragma unroll
                for (int j = 0; j < 2; ++j) zl[j * THREADS] = make_double2(acc[0][j][0], acc[0][j][1]);
            }
            if (l + 1 < L) {
#pragma unroll
                for (int s = 0; s < S; ++s)
#pragma unroll
                    for (int j = 0; j < 2; ++j)
                        *reinterpret_cast<double2*>(act + (s * TP + g) * LD + col0 + 8 * j + 2 * t) =
                            make_double2(acc[s][j][0], acc[s][j][1]);
                if (backward) asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            }
        }

        // ------------------------- head and residual -------------------------
        double wh[2][2];
#pragma unroll
        for (int j = 0; j < 2; ++j)
#pragma unroll
            for (int c = 0; c < 2; ++c) wh[j][c] = phead[unit_of(j, c)];
#pragma unroll
        for (int s = 0; s < S; ++s) {
            double dot = 0.0;
#pragma unroll
            for (int j = 0; j < 2; ++j) dot += acc[s][j][0] * wh[j][0] + acc[s][j][1] * wh[j][1];
            dot += __shfl_xor_sync(0xffffffffu, dot, 1);
            dot += __shfl_xor_sync(0xffffffffu, dot, 2);
            if (t == 0) red[(warp * S + s) * TP + g] = dot;
        }
        __syncthreads();
        if (tid < TP) {
            const long long p = p0 + tid;
            const bool valid = p < a.n_points;
            const long long pc = valid ? p : a.n_points - 1;
#pragma unroll
            for (int s = 0; s < S; ++s) {
                double u = red[s * TP + tid];
#pragma unroll
                for (int q = 1; q < NW; ++q) u += red[(q * S + s) * TP + tid];
                us[s * TP + tid] = s == 0 ? u + head_bias : u;
            }
            double r[MAX_REGS];
            run_program<double>(code, a.prog.n_instr, static_cast<const double*>(a.prog.consts), a.table + pc * a.ncols,
                                us + tid, TP, r);
            if (valid) loss_sum += r[a.prog.value_reg];
#pragma unroll
            for (int s = 0; s < S; ++s) {
                const int reg = a.prog.grad_regs[s];
                uh[s * TP + tid] = (valid && reg >= 0) ? seed * r[reg] : 0.0;
            }
        }
        __syncthreads();
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
            double pw[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll
            for (int s = 0; s < S; ++s) {
                const double u = uh[s * TP + g];
#pragma unroll
                for (int j = 0; j < 2; ++j)
#pragma unroll
                    for (int c = 0; c < 2; ++c) {
                        pw[2 * j + c] += acc[s][j][c] * u;
                        acc[s][j][c] = u * wh[j][c];
                    }
            }
            add_column_sums64(pw, ghead, lane, col0, t);
            if (tid == 0) {
                double total = 0.0;
#pragma unroll
                for (int p = 0; p < TP; ++p) total += uh[p];
                head_bias_grad += total;
            }
        }
        for (int l = L - 1; l >= 0; --l) {
            const double2* zl = reinterpret_cast<const double2*>(sz + (size_t)l * G::SCRATCH_PER_CTA) + tid;
#pragma unroll
            for (int j = 0; j < 2; ++j) {
                double z[S][2];
#pragma unroll
                for (int s = 0; s < S; ++s) {
                    const double2 q = zl[(2 * s + j) * THREADS];
                    z[s][0] = q.x;
                    z[s][1] = q.y;
                }
#pragma unroll
                for (int c = 0; c < 2; ++c) {
                    double zc[S], gc[S];
#pragma unroll
                    for (int s = 0; s < S; ++s) {
                        zc[s] = z[s][c];
                        gc[s] = acc[s][j][c];
                    }
                    if (ACT == ACT_TANH)
                        jet_apply_transposed_with<double, SG>(TanhD<double>(zc[0]), zc, gc, a.merge_w);
                    else
                        jet_apply_transposed<double, SG, ACT>(zc, gc, a.merge_w);
#pragma unroll
                    for (int s = 0; s < S; ++s) acc[s][j][c] = gc[s];
                }
            }
            {
                double pb[4] = {acc[0][0][0], acc[0][0][1], acc[0][1][0], acc[0][1][1]};
                add_column_sums64(pb, gbias + l * W, lane, col0, t);
            }
            if (l == 0) {
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    if (k < d0) {
                        double pw[4];
#pragma unroll
                        for (int j = 0; j < 2; ++j)
#pragma unroll
                            for (int c = 0; c < 2; ++c) {
                                double v = x[k] * acc[0][j][c];
#pragma unroll
                                for (int dj = 0; dj < SG::ndirs; ++dj) v += a.dirs[dj * d0 + k] * acc[SG::base(dj)][j][c];
                                pw[2 * j + c] = v;
                            }
                        add_column_sums64(pw, gfirst + k * W, lane, col0, t);
                    }
                }
                break;
            }
            // Cotangents of the pre-activations: operand of both contractions below.
#pragma unroll
            for (int s = 0; s < S; ++s)
#pragma unroll
                for (int j = 0; j < 2; ++j)
                    *reinterpret_cast<double2*>(act + (s * TP + g) * LD + col0 + 8 * j + 2 * t) =
                        make_double2(acc[s][j][0], acc[s][j][1]);
            mbar_wait(hbar, hphase, a.error);
            hphase ^= 1;
            __syncthreads();
            // Weight gradient: dW[k][n] += sum_rows H[row][k] * Zhat[row][n]; this warp: its 16 k x all n, 16 n at a time.
            {
                double2* gw = dws + (size_t)(l - 1) * 4 * NW * THREADS + tid;
                const double* a_lane = ht + t * LD + col0 + g;
                const double* b_lane = act + t * LD + g;
#pragma unroll
                for (int nb = 0; nb < NW; ++nb) {
                    double dw[2][2][2];
#pragma unroll
                    for (int m = 0; m < 2; ++m)
#pragma unroll
                        for (int j = 0; j < 2; ++j) {
                            const double2 q = gw[(4 * nb + 2 * m + j) * THREADS];
                            dw[m][j][0] = q.x;
                            dw[m][j][1] = q.y;
                        }
#pragma unroll
                    for (int k = 0; k < S * TP; k += 4) {
                        const double a0 = a_lane[k * LD], a1 = a_lane[k * LD + 8];
                        const double b0 = b_lane[k * LD + nb * 16], b1 = b_lane[k * LD + nb * 16 + 8];
                        dmma_m8n8k4(dw[0][0], a0, b0);
                        dmma_m8n8k4(dw[0][1], a0, b1);
                        dmma_m8n8k4(dw[1][0], a1, b0);
                        dmma_m8n8k4(dw[1][1], a1, b1);
                    }
#pragma unroll
                    for (int m = 0; m < 2; ++m)
#pragma unroll
                        for (int j = 0; j < 2; ++j) gw[(4 * nb + 2 * m + j) * THREADS] = make_double2(dw[m][j][0], dw[m][j][1]);
                }
            }
            // Cotangents of layer l-1's jets: G = Zhat W^T.
            mbar_wait(wbar, wphase, a.error);
            wphase ^= 1;
            warp_contract64<S, W, LD, false>(act, wbuf, warp, g, t, acc);
            __syncthreads();
            if (tid == 0) {
                load_weights();
                if (l > 1) load_jets(l - 2);
            }
        }
    }

    // Per-CTA gradients in parameter order, and the loss partial, in a fixed order.
    __syncthreads();
    if (backward) {
        double* my_grad = a.grad_cta + (size_t)blockIdx.x * a.P;
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
            double* out = my_grad + a.w_off[l];
            for (int q = 0; q < 4 * NW; ++q) {
                const double2 v = dws[((size_t)(l - 1) * 4 * NW + q) * THREADS + tid];
                const int k = col0 + ((q >> 1) & 1) * 8 + g, n = (q >> 2) * 16 + (q & 1) * 8 + 2 * t;
                if (k < rows && n < cols) out[k * cols + n] = v.x;
                if (k < rows && n + 1 < cols) out[k * cols + n + 1] = v.y;
            }
        }
    }
    if (tid < TP) red[tid] = loss_sum;
    __syncthreads();
    if (tid == 0) {
        double total = 0.0;
        for (int p = 0; p < TP; ++p) total += red[p];
        a.loss_cta[blockIdx.x] = total;
    }
}

}  // namespace qb
