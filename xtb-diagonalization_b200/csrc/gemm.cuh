// Grouped GEMM for the eigensolver's matrix-shaped stages (sm_100a).
//
//   C_p = alpha_p op(A_p) op(B_p) + beta_p C_p      for every problem p of a group, in one launch
//
// Column-major operands, as LAPACK/BLAS.  FP64 runs on the double-precision tensor pipe (mma.sync m8n8k4 f64);
// FP32 uses the same tiling with CUDA-core FMAs (the FP32 path is the ssytrd/sormtr ABI, which must keep FP32
// rounding, so it does not use TF32).
//
// Triangular operands are masked per element, so the unused triangle of a stored matrix may hold anything:
//   kTriAUpper: op(A)(m,k) = 0 for k < m      kTriALower: op(A)(m,k) = 0 for k > m
//   kTriBUpper: op(B)(k,n) = 0 for k > n      kTriBLower: op(B)(k,n) = 0 for k < n
// and the K loop of each output tile is clipped to the nonzero band.  kCUpper skips output tiles strictly below the
// diagonal (their C is left untouched).
//
// Descriptors live in device memory, so a kernel may write a problem's sizes before the GEMM runs (the divide and
// conquer merges know their sizes only on the device).  The host fixes each problem's tile grid (tiles_m, tiles_n)
// from an upper bound; tiles outside the actual M x N return at once.
#pragma once
#include <cuda_runtime.h>

namespace xtbeig {

enum GemmMode : int {
  kTriAUpper = 1,
  kTriALower = 2,
  kTriBUpper = 4,
  kTriBLower = 8,
  kCUpper = 16,
};

template <typename T>
struct GemmDesc {
  const T* A;
  const T* B;
  T* C;
  int M, N, K;
  int lda, ldb, ldc;
  T alpha, beta;
  int transA, transB;
  int mode;
  int tile_begin;  // first global tile index of this problem
  int tiles_m, tiles_n;
};

constexpr int kGemmBM = 64, kGemmBN = 64, kGemmBK = 16, kGemmThreads = 128;
constexpr int kGemmInlineMax = 32;  // descriptors passed by value in the launch (parameter space)

inline long gemm_tiles(int m, int n, int edge) { return (long)((m + edge - 1) / edge) * ((n + edge - 1) / edge); }

// Edge of the output tiles of a launch whose problems have tiles64 tiles of 64 x 64, or tiles32 of 32 x 32, together.  The
// cost of a K step (16) on the busiest of the 148 SMs, in units of a 32 x 32 tile (FP64 0.24 us, FP32 0.30): one, two,
// three 64 x 64 tiles together take 4.4, 5.6, 8.5 units (FP64: 1.05, 1.32, 2.0 us; a lone CTA waits for its own loads and
// products), or 3.5, 4.4, 6.3 (FP32); a fourth waits for a place; 32 x 32 tiles take 1 each.  So 32 x 32 wins up to about
// 200 tiles of 64 x 64 (FP32: 100), and where a few tiles would start a second wave.  FP64: 412^3 16.5 us against 28.8,
// 130^3 6.2 / 12.3, 840^3 57 / 70, 1350^3 222 / 269; but 940^3 85 / 78, 1788^3 465 / 425.
template <typename T>
int gemm_tile_edge(long tiles64, long tiles32) {
  constexpr bool f64 = sizeof(T) == 8;
  const double cost[3] = {f64 ? 4.4 : 3.5, f64 ? 5.6 : 4.4, f64 ? 8.5 : 6.3};
  const long slots = 3 * 148, rest = tiles64 % slots;
  const double c64 = (double)(tiles64 / slots) * cost[2] + (rest > 0 ? cost[(rest - 1) / 148] : 0.0);
  return (double)((tiles32 + 147) / 148) < c64 ? 32 : 64;
}

// Launch a group: descs (device) holds nprob descriptors whose tiles_m, tiles_n count tiles of `edge` and whose
// tile_begin are their prefix sum; total_tiles their sum.  Returns the launch's error, which no later call reports.
template <typename T>
cudaError_t gemm_grouped_launch(const GemmDesc<T>* d_descs, int nprob, int total_tiles, int edge, cudaStream_t s);

}  // namespace xtbeig
