// Compact-WY helpers shared by the back-transformations (ormtr after the one-stage reduction, Q1 after sy2sb):
// the forward T factor of a block of reflectors from its Gram matrix, and the ordered sum of split-K partial products.
#pragma once
#include <algorithm>

#include "gemm_tile.cuh"
#include "kernels.h"

namespace xtbeig {
namespace {

constexpr int kMaxSplit = 8;  // split-K slices at most (Gram matrices, ormtr's W = V^T Z)

// Split-K slices of the Gram matrix G_b = V_b^T V_b of a block whose reflectors reach `rows` rows: slices of at
// least 128 rows, at most `S`.  The host's GEMMs and wy_factor_kernel's loader use the same count.
__host__ __device__ inline int gram_slices(int rows, int S) { return max(1, min(S, rows / 128)); }

// The upper-triangular forward factor T_b of each block of reflectors (one CTA per block):
//   H_j0 ... H_j1 = I - V_b T_b V_b^T,   T(i,i) = tau_i,   T(0:i-1, i) = -tau_i T(0:i-1, 0:i-1) G(0:i-1, i).
// G_b = V_b^T V_b arrives as S_b = gram_slices(rows_b, S) split-K partial products (kb x kb, ld nb, slice stride
// nb * nb, block stride S * nb * nb) that the loader sums in slice order; T_b leaves in tf (ld nb).  The factor is
// built in shared memory by blocks: diagonal blocks of at most 16 by the column recurrence (one warp each), then
// neighbours of s = 16, 32, 64, ... columns are joined, since for V = [V1 V2]
//   (I - V1 T1 V1^T)(I - V2 T2 V2^T) = I - V [[T1, -T1 G12 T2], [0, T2]] V^T.
// G's strict upper triangle is kept transposed in the strict lower triangle of the same array.  M = G12 T2 goes where T12
// will be; -T1 M goes where G12 was (nothing reads it again) and is then copied over M.  Both products run on 8 x 8 tiles
// of the FP64 tensor pipe (an FP32 block too: its entries are widened, so its sums only gain), a warp per tile.  The
// recurrence is sequential only inside the diagonal blocks.  What bounds it: the latency of the chain of joins on one SM; a
// kernel that formed T12's rows one after another and divided for every index took 159 us for 14 blocks of 128 (two
// blocks: 115), now 50 (22).
// The leading dimension nb + kWyPad puts the 4 x 8 elements of a tile's operand on different banks.
constexpr int kWyThreads = 512;

template <typename T>
__global__ void __launch_bounds__(kWyThreads) wy_factor_kernel(int nm1, int nb, const T* __restrict__ tau,
                                                        const T* __restrict__ parts, int S, T* __restrict__ tf) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  // nb x nb: T (upper with diagonal), G transposed (strict lower)
  const int ld = nb + kWyPad;
  T* Ts = reinterpret_cast<T*>(smem_raw);
  T* ts = Ts + (size_t)nb * ld;  // tau of the block
  const int b = blockIdx.x, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nwarp = blockDim.x >> 5;
  const int j0 = b * nb;
  const int kb = min(nb, nm1 - j0);
  const int Sb = gram_slices(j0 + kb, S);
  const T* gp = parts + (size_t)b * S * nb * nb;
  // A warp per column, up to four rows per lane and every slice of them in flight at once (the partial products come from
  // L2); slices are added in order.
  constexpr int U = 4;
  const size_t slice = (size_t)nb * nb;
  for (int c = warp; c < kb; c += nwarp) {
    for (int r0 = lane; r0 < c; r0 += 32 * U) {
      const T* gc = gp + r0 + (size_t)c * nb;  // G(r0, c)
      T v[U] = {};
#pragma unroll
      for (int sl = 0; sl < kMaxSplit; ++sl) {
        if (sl >= Sb) break;
#pragma unroll
        for (int u = 0; u < U; ++u)
          if (r0 + 32 * u < c) v[u] += gc[32 * u];
        gc += slice;
      }
#pragma unroll
      for (int u = 0; u < U; ++u)
        if (r0 + 32 * u < c) Ts[c + (r0 + 32 * u) * ld] = v[u];  // stored at (c, r)
    }
  }
  for (int i = tid; i < kb; i += blockDim.x) ts[i] = tau[j0 + i];
  __syncthreads();
  auto G = [&](int r, int c) { return Ts[c + (size_t)r * ld]; };  // G(r, c), r < c
  // Diagonal blocks of at most 16: lane r keeps row r of T in registers, so a column waits only for its own lane's last
  // entry; G(c, i) is the same for every lane.
  for (int o = warp * 16; o < kb; o += nwarp * 16) {
    const int L = min(16, kb - o);
    T t[16];
#pragma unroll
    for (int i = 0; i < 16; ++i) {
      T acc0 = T(0), acc1 = T(0);
      if (i < L) {
#pragma unroll
        for (int c = 0; c < i; ++c) {
          if (c & 1) acc1 = fma(t[c], G(o + c, o + i), acc1);
          else acc0 = fma(t[c], G(o + c, o + i), acc0);
        }
      }
      const T ti = i < L ? ts[o + i] : T(0);
      t[i] = lane == i ? ti : lane < i ? -ti * (acc0 + acc1) : T(0);
    }
#pragma unroll
    for (int i = 0; i < 16; ++i)
      if (i < L && lane <= i) Ts[(o + lane) + (size_t)(o + i) * ld] = t[i];
  }
  __syncthreads();
  const int g = lane >> 2, l4 = lane & 3;
  for (int lg = 4; (1 << lg) < kb; ++lg) {
    const int s = 1 << lg;
    // Pair p joins columns o .. o + s - 1 and c0 = o + s .. (o = 2 s p); its tiles of 8 x 8 are numbered column by
    // column.  A tile's columns past the block's end are computed from its last column and not stored.
    const int pairs = (kb - s + 2 * s - 1) >> (lg + 1), tiles = pairs << 2 * (lg - 3);
    // M(r, c) = sum_{q <= c} G12(r, q) T2(q, c).
    for (int t = warp; t < tiles; t += nwarp) {
      const int o = (t >> 2 * (lg - 3)) << (lg + 1), c0 = o + s, n2 = kb - c0;
      const int r = (t & ((s >> 3) - 1)) * 8 + g, tc = ((t >> (lg - 3)) & ((s >> 3) - 1)) * 8;
      if (tc >= n2) continue;
      const int kend = min(tc + 8, n2), c = min(tc + g, n2 - 1);
      const T* pa = Ts + c0 + (o + r) * ld;
      const T* pb = Ts + c0 + (c0 + c) * ld;
      double acc[2][2] = {{0, 0}, {0, 0}};
#pragma unroll 2
      for (int k0 = 0; k0 < kend; k0 += 8)
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const int k = min(k0 + 4 * h + l4, n2 - 1);
          const double a = (double)pa[k], bv = (double)pb[k];
          tile::mma_f64(acc[h], a, k0 + 4 * h + l4 <= c ? bv : 0.0);
        }
#pragma unroll
      for (int i = 0; i < 2; ++i)
        if (tc + 2 * l4 + i < n2) Ts[(o + r) + (c0 + tc + 2 * l4 + i) * ld] = (T)(acc[0][i] + acc[1][i]);
    }
    __syncthreads();
    // T12(r, c) = -sum_{q >= r} T1(r, q) M(q, c), into (c0 + c, o + r).
    for (int t = warp; t < tiles; t += nwarp) {
      const int o = (t >> 2 * (lg - 3)) << (lg + 1), c0 = o + s, n2 = kb - c0;
      const int tr = (t & ((s >> 3) - 1)) * 8, r = tr + g, tc = ((t >> (lg - 3)) & ((s >> 3) - 1)) * 8;
      if (tc >= n2) continue;
      const T* pa = Ts + (o + r) + (o + l4) * ld;
      const T* pb = Ts + (o + l4) + (c0 + min(tc + g, n2 - 1)) * ld;
      double acc[2][2] = {{0, 0}, {0, 0}};
#pragma unroll 2
      for (int k0 = tr; k0 < s; k0 += 8)
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const double a = (double)pa[(k0 + 4 * h) * ld], bv = (double)pb[k0 + 4 * h];
          tile::mma_f64(acc[h], k0 + 4 * h + l4 >= r ? a : 0.0, bv);
        }
#pragma unroll
      for (int i = 0; i < 2; ++i)
        if (tc + 2 * l4 + i < n2) Ts[(c0 + tc + 2 * l4 + i) + (o + r) * ld] = (T)(-(acc[0][i] + acc[1][i]));
    }
    __syncthreads();
    for (int c = warp; c < kb; c += nwarp)
      if ((c >> lg) & 1)
        for (int r = ((c >> lg) - 1) * s + lane; r < (c >> lg) * s; r += 32) Ts[r + c * ld] = Ts[c + r * ld];
    __syncthreads();
  }
  T* tb = tf + (size_t)b * nb * nb;
  for (int c = warp; c < kb; c += nwarp)
    for (int r = lane; r < kb; r += 32) tb[r + (size_t)c * nb] = r <= c ? Ts[r + c * ld] : T(0);
}

// W = sum over the split-K slices, in slice order (deterministic): parts is S slices of kb x m (ld nb, stride nb*m).
template <typename T>
__global__ void splitk_sum_kernel(int kb, int m, int nb, int S, const T* __restrict__ parts, T* __restrict__ w) {
  const size_t total = (size_t)kb * m;
  const size_t stride = (size_t)nb * m;
  for (size_t idx = (size_t)blockIdx.x * blockDim.x + threadIdx.x; idx < total; idx += (size_t)gridDim.x * blockDim.x) {
    const int r = (int)(idx % kb), c = (int)(idx / kb);
    const size_t off = r + (size_t)c * nb;
    T acc = parts[off];
    for (int sl = 1; sl < S; ++sl) acc += parts[off + sl * stride];
    w[off] = acc;
  }
}

// Split-K slices for W = V_b^T Z: enough CTAs to cover the SMs twice, slices of at least 128 rows.
inline int split_count(int kb, int m, int rows, int bm = kGemmBM, int bn = kGemmBN) {
  const int tiles = ((kb + bm - 1) / bm) * ((m + bn - 1) / bn);
  int S = (2 * 148 + tiles - 1) / tiles;
  S = std::min(S, std::max(1, rows / 128));
  return std::max(1, std::min(S, kMaxSplit));
}

}  // namespace
}  // namespace xtbeig
