// One BT x BT output tile (64 or 32) of C = alpha op(A) op(B) + beta C computed by a whole CTA of kGemmThreads (4 warps
// of BT/2 x BT/2).  Shared by the grouped GEMM kernel and by the persistent Cholesky kernel, which calls it from inside
// its own phases.  FP64 issues mma.sync.m8n8k4 f64 (layout of the PTX ISA's m8n8k4 .f64 shape: A row = lane/4,
// col = lane%4; B row = lane%4, col = lane/4; C row = lane/4, cols 2*(lane%4) + {0,1}); FP32 uses CUDA-core FMAs on
// the same tiling (the FP32 ABI must keep FP32 rounding).  K runs through a STAGES-deep cp.async pipeline.
//
// What bounds it: with one CTA per SM (small problems) the latency of a K step, with three the FP64 pipe.  A thread's
// source pointers are formed once per tile and stepped along K, and the tests for the matrix's edge and the triangles
// are made only in the K steps that need them: formed per element, the addresses took longer than the step's
// multiplications (a lone CTA 1.9 us per step of 16, now 1.05; 1788^3 at 20.9 TFLOP/s, now 26.9).  Tiles of 32 x 32
// spread a small problem over four times as many SMs (gemm_tile_edge).
#pragma once
#include <cuda_runtime.h>

#include "gemm.cuh"

namespace xtbeig {
namespace tile {

constexpr int BK = kGemmBK;
// Three K-tiles in flight while one is consumed hides L2/HBM latency behind the DMMA loop.
constexpr int STAGES = 4;

// smem row stride (elements) of a K-tile: 4 (mod 16) keeps each half-warp's fragment loads on 16 distinct 8-byte banks.
template <int BT>
constexpr int kStride = BT + 4;

template <typename T, int BT = kGemmBM>
constexpr size_t smem_elems() {
  return (size_t)STAGES * 2 * BK * kStride<BT>;
}

__device__ __forceinline__ void cp_async_8(void* smem, const void* gmem, bool pred) {
  unsigned s = (unsigned)__cvta_generic_to_shared(smem);
  int sz = pred ? 8 : 0;
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(s), "l"(gmem), "r"(sz) : "memory");
}
__device__ __forceinline__ void cp_async_4(void* smem, const void* gmem, bool pred) {
  unsigned s = (unsigned)__cvta_generic_to_shared(smem);
  int sz = pred ? 4 : 0;
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(s), "l"(gmem), "r"(sz) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

template <typename T>
__device__ __forceinline__ void cp_elem(T* smem, const T* gmem, bool pred);
template <>
__device__ __forceinline__ void cp_elem<double>(double* smem, const double* gmem, bool pred) {
  cp_async_8(smem, gmem, pred);
}
template <>
__device__ __forceinline__ void cp_elem<float>(float* smem, const float* gmem, bool pred) {
  cp_async_4(smem, gmem, pred);
}

// One operand's share of a thread: element i of a K-tile is (row r + i dr, k kk + i dk) of the operand seen as rows x K
// (op(A)'s rows or op(B)'s columns), with the smaller index running along memory.
template <typename T, int BT>
struct Loader {
  static constexpr int E = BT * BK / kGemmThreads;
  const T* ptr;        // element 0 of K-tile 0 (k = klo)
  size_t step;         // elements between consecutive i
  size_t advance;      // elements per K-tile
  int r, kk, dr, dk;   // element 0's row (within the tile) and k (within the K-tile), and their steps

  // along_k: k runs along memory (transposed A, plain B).
  __device__ __forceinline__ void init(const T* base, int ld, bool along_k, int r0, int klo) {
    const int tid = threadIdx.x;
    if (along_k) {
      // Half a warp takes 4 rows x 4 k: 16 distinct banks of the transposed K-tile, whole sectors of memory.
      kk = (tid & 3) | ((tid >> 2) & 12);
      r = ((tid >> 2) & 3) | ((tid >> 4) & ~3);
      dr = kGemmThreads / BK;
      dk = 0;
      ptr = base + (klo + kk) + (size_t)(r0 + r) * ld;
      step = (size_t)dr * ld;
      advance = BK;
    } else {
      r = tid % BT;
      kk = tid / BT;
      dr = 0;
      dk = kGemmThreads / BT;
      ptr = base + (r0 + r) + (size_t)(klo + kk) * ld;
      step = (size_t)dk * ld;
      advance = (size_t)BK * ld;
    }
  }
  // The K-tile at k0 (kt tiles after klo) into dst[k][row].  full: every element lies in the matrix and the kept
  // triangle.  keep_ge / keep_le: only k >= row / k <= row.  An element that is not loaded is zero-filled (source size 0).
  __device__ __forceinline__ void load(T* dst, const T* base, int kt, int k0, int r0, int R, int K, bool full,
                                       bool keep_ge, bool keep_le) const {
    const T* src = ptr + (size_t)kt * advance;
    T* d = dst + kk * kStride<BT> + r;
    const int dstep = dk * kStride<BT> + dr;
    if (full) {
#pragma unroll
      for (int i = 0; i < E; ++i) cp_elem<T>(d + i * dstep, src + i * step, true);
    } else {
#pragma unroll
      for (int i = 0; i < E; ++i) {
        const int gr = r0 + r + i * dr, gk = k0 + kk + i * dk;
        bool ok = gr < R && gk < K;
        if (keep_ge) ok = ok && gk >= gr;
        if (keep_le) ok = ok && gk <= gr;
        cp_elem<T>(d + i * dstep, ok ? src + i * step : base, ok);
      }
    }
  }
};

__device__ __forceinline__ void mma_f64(double (&c)[2], double a, double b) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};"
               : "+d"(c[0]), "+d"(c[1])
               : "d"(a), "d"(b));
}

template <typename T, int MI, int ST>
struct Frag;

template <int MI, int ST>
struct Frag<double, MI, ST> {
  __device__ __forceinline__ static void step(double (&acc)[MI][MI][2], const double* As, const double* Bs, int kk,
                                              int wm, int wn, int lane) {
    double a[MI], b[MI];
    const int kr = kk * 4 + (lane & 3), g = lane >> 2;
#pragma unroll
    for (int i = 0; i < MI; ++i) a[i] = As[kr * ST + wm * MI * 8 + i * 8 + g];
#pragma unroll
    for (int j = 0; j < MI; ++j) b[j] = Bs[kr * ST + wn * MI * 8 + j * 8 + g];
#pragma unroll
    for (int i = 0; i < MI; ++i)
#pragma unroll
      for (int j = 0; j < MI; ++j) mma_f64(acc[i][j], a[i], b[j]);
  }
};

template <int MI, int ST>
struct Frag<float, MI, ST> {
  __device__ __forceinline__ static void step(float (&acc)[MI][MI][2], const float* As, const float* Bs, int kk,
                                              int wm, int wn, int lane) {
    const int g = lane >> 2, c2 = (lane & 3) * 2;
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const int kr = kk * 4 + q;
      float a[MI], b0[MI], b1[MI];
#pragma unroll
      for (int i = 0; i < MI; ++i) a[i] = As[kr * ST + wm * MI * 8 + i * 8 + g];
#pragma unroll
      for (int j = 0; j < MI; ++j) {
        b0[j] = Bs[kr * ST + wn * MI * 8 + j * 8 + c2];
        b1[j] = Bs[kr * ST + wn * MI * 8 + j * 8 + c2 + 1];
      }
#pragma unroll
      for (int i = 0; i < MI; ++i)
#pragma unroll
        for (int j = 0; j < MI; ++j) {
          acc[i][j][0] = fmaf(a[i], b0[j], acc[i][j][0]);
          acc[i][j][1] = fmaf(a[i], b1[j], acc[i][j][1]);
        }
    }
  }
};

// The tile at (m0, n0) of problem p, by all kGemmThreads threads of the CTA.  smem holds smem_elems<T, BT>() elements.
// Returns after a __syncthreads, so the caller may reuse smem at once.  Tiles wholly outside C, or below the diagonal
// under kCUpper, return without touching memory (uniformly for the CTA).
template <typename T, int BT = kGemmBM>
__device__ void gemm_tile(const GemmDesc<T>& p, int m0, int n0, T* smem) {
  constexpr int MI = BT / 16, ST = kStride<BT>, KT = BK * ST;
  if (m0 >= p.M || n0 >= p.N) return;
  if ((p.mode & kCUpper) && m0 > n0 + BT - 1) return;
  T* As = smem;                // [STAGES][BK][ST]
  T* Bs = As + STAGES * KT;    // [STAGES][BK][ST]
  const int mode = p.mode;
  int klo = 0, khi = p.K;
  if (mode & kTriAUpper) klo = max(klo, m0);
  if (mode & kTriBLower) klo = max(klo, n0);
  if (mode & kTriALower) khi = min(khi, m0 + BT);
  if (mode & kTriBUpper) khi = min(khi, n0 + BT);
  klo = (klo / BK) * BK;

  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int wm = warp & 1, wn = warp >> 1;
  T acc[MI][MI][2];
#pragma unroll
  for (int i = 0; i < MI; ++i)
#pragma unroll
    for (int j = 0; j < MI; ++j) acc[i][j][0] = acc[i][j][1] = T(0);

  const int nk = khi > klo ? (khi - klo + BK - 1) / BK : 0;
  if (nk > 0) {
    Loader<T, BT> la, lb;
    la.init(p.A, p.lda, p.transA != 0, m0, klo);
    lb.init(p.B, p.ldb, p.transB == 0, n0, klo);
    const bool fit_a = m0 + BT <= p.M, fit_b = n0 + BT <= p.N;
    auto load = [&](int kt, int buf) {
      const int k0 = klo + kt * BK;
      const bool fit_k = k0 + BK <= p.K;
      // A K-tile wholly on the kept side of a triangle needs no test.
      const bool a_ge = (mode & kTriAUpper) && k0 < m0 + BT - 1, a_le = (mode & kTriALower) && k0 + BK - 1 > m0;
      const bool b_le = (mode & kTriBUpper) && k0 + BK - 1 > n0, b_ge = (mode & kTriBLower) && k0 < n0 + BT - 1;
      la.load(As + buf * KT, p.A, kt, k0, m0, p.M, p.K, fit_a && fit_k && !a_ge && !a_le, a_ge, a_le);
      lb.load(Bs + buf * KT, p.B, kt, k0, n0, p.N, p.K, fit_b && fit_k && !b_ge && !b_le, b_ge, b_le);
    };
#pragma unroll 1
    for (int st = 0; st < STAGES - 1; ++st) {
      if (st < nk) load(st, st);
      cp_async_commit();
    }
    int cur = 0;
#pragma unroll 1
    for (int it = 0; it < nk; ++it) {
      cp_async_wait<STAGES - 2>();  // K-tile `it` has landed
      __syncthreads();              // ... for every thread, and K-tile it-1's buffer is free
      const int pf = it + STAGES - 1;
      if (pf < nk) load(pf, (cur + STAGES - 1) % STAGES);
      cp_async_commit();
#pragma unroll
      for (int kk = 0; kk < BK / 4; ++kk)
        Frag<T, MI, ST>::step(acc, As + cur * KT, Bs + cur * KT, kk, wm, wn, lane);
      cur = (cur + 1) % STAGES;
    }
    cp_async_wait<0>();
  }
  __syncthreads();  // every warp is done with smem (the caller may reuse it) and has read its A/B data

  const T alpha = p.alpha, beta = p.beta;
  const int g = lane >> 2, c2 = (lane & 3) * 2;
  // Every read of C before the first write: they are the same addresses, but the compiler cannot tell the elements apart.
  if (beta != T(0)) {
#pragma unroll
    for (int i = 0; i < MI; ++i)
#pragma unroll
      for (int j = 0; j < MI; ++j)
#pragma unroll
        for (int c = 0; c < 2; ++c) {
          const int gm = m0 + wm * MI * 8 + i * 8 + g, gn = n0 + wn * MI * 8 + j * 8 + c2 + c;
          const bool in = gm < p.M && gn < p.N && !((mode & kCUpper) && gm > gn);
          const T old = in ? p.C[gm + (size_t)gn * p.ldc] : T(0);
          acc[i][j][c] = alpha * acc[i][j][c] + beta * old;
        }
  } else {
#pragma unroll
    for (int i = 0; i < MI; ++i)
#pragma unroll
      for (int j = 0; j < MI; ++j)
#pragma unroll
        for (int c = 0; c < 2; ++c) acc[i][j][c] *= alpha;
  }
#pragma unroll
  for (int i = 0; i < MI; ++i) {
    const int gm = m0 + wm * MI * 8 + i * 8 + g;
#pragma unroll
    for (int j = 0; j < MI; ++j)
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        const int gn = n0 + wn * MI * 8 + j * 8 + c2 + c;
        if (gm < p.M && gn < p.N && !((mode & kCUpper) && gm > gn))  // kCUpper updates the upper triangle only
          p.C[gm + (size_t)gn * p.ldc] = acc[i][j][c];
      }
  }
}

}  // namespace tile
}  // namespace xtbeig
