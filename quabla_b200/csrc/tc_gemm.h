// Launchers of the tcgen05 float32 GEMMs (tc_tma_gemm.cuh).
#pragma once
#include <cuda_runtime.h>

#include <cstddef>
#include <cstdint>

namespace qb {

// Shapes the tensor-core kernels accept.
bool tc_rows_ok(int N, int K);     // C[M][N] = A[M][K] * W: N % 64 == 0, 64 <= N <= 256, K % 32 == 0
bool tc_wgrad_ok(int Mw, int N);   // P = H^T G with H [rows][Mw], G [rows][N]: Mw % 128 == 0, N as above
// Whether the tensor-core GEMMs can run: QB200_TC=0 switches them off, and the driver must provide the
// tensor-map encoder (operands arrive by TMA tensor maps).
bool tc_available();
// How the forward and data-gradient GEMMs split float32 operands (tc_tma_gemm.cuh); tc_scheme() is TC_F16 unless
// QB200_TC_COR=tf32|bf16 asks for another.
enum TcScheme { TC_TF32, TC_BF16, TC_F16 };
TcScheme tc_scheme();

// float32 words of the per-layer weight image of a weight [K][N] (tc2_prepare_launch), four parts of K*N words:
//   TC_F16   [pair matrix of W^T | pair matrix of W | factors of the N rows of W^T, then of the K rows of W | unused]
//   TC_BF16  [tf32(W^T) | pair matrix of W^T | pair matrix of W | tf32(W)]
//   TC_TF32  [W^T | lo(W^T) | lo(W) | unused]
// A pair matrix holds per row and per 32 contraction elements 32 first parts (f16 hi, or bf16(v)) then 32 second ones
// (f16 lo, or bf16(v - tf32(v))), i.e. 128-byte rows that one tensor-map box brings per k-tile.
size_t tc_image_words(int K, int N);
struct TcImage { float *first, *second, *third, *fourth; };
TcImage tc_image(float* words, int K, int N);

// Writes the image of W [K][N] into `words`.
cudaError_t tc2_prepare_launch(const float* w, int K, int N, float* words, TcScheme scheme, cudaStream_t stream);
// C = A W (forward, A [M][K], + bias on the first bias_rows rows) or C = A W^T (dgrad, A [M][N]) with the image that
// tc2_prepare_launch wrote for W [K][N] under the same scheme.
cudaError_t tc2_rows_launch(const float* A, int M, int K, int N, const float* w, float* words, bool dgrad, float* C,
                            const float* bias, int bias_rows, TcScheme scheme, int* error, cudaStream_t stream);
cudaError_t tc2_wgrad_launch(const float* H, int ldh, const float* G, int ldg, float* partials, int rows, int Mw, int N,
                             int rows_per_slice, int* error, cudaStream_t stream);

}  // namespace qb
