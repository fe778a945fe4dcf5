// One-stage reduction to tridiagonal form, LAPACK xsytrd semantics with UPLO = 'U' (the contract of xtb_dsytrd_upper,
// reference Sources/Diagonalization/Exports.swift:8-27; LAPACK dlatrd/dsytd2 order as in Tridiagonalization.swift
// :511-618): for k = n-1 ... 1 (0-based) the reflector H(k-1) = I - tau v v^T annihilates A(0:k-2, k) against
// A(k-1, k); v(k-1) = 1, v(0:k-2) is stored in A(0:k-2, k), e(k-1) = beta, and A(0:k-1, 0:k-1) <- H A H.
//
// B200 design (not a port of the reference's blocked CPU code).  The reduction is a chain of n-1 dependent
// matrix-vector products, so on a GPU its cost is the grid-wide dependency per column, not flops.  One persistent
// cooperative kernel keeps the whole symmetric matrix on chip: rows are dealt to the CTAs in small blocks, cyclically
// (so the shrinking trailing matrix stays balanced); a CTA's first RR rows live in registers (thread t holds the column
// pairs 2(t + j NT), + 1 of them), the others in shared memory or, when they do not fit, in a global (L2-resident) slab.
// Per column k every CTA
//   1. holds x = A(0:k-1, k) in registers (the columns of thread t) and in shared memory;
//   2. in ONE pass over its own rows applies the previous step's rank-2 update A -= v w^T + w v^T and accumulates
//      (A x)_r with x itself rather than v: v = (scale x(0:k-2), 1), so y = A v = scale (A x)_r + A(r, k-1), and
//      the Householder scalars are not needed before the pass (the update of step k+1 fused with the symv of step k);
//      the previous w at own rows is formed from the previous y and v at own rows, w = tau y - tau^2/2 (y.v) v, as
//      the owner of each column forms it;
//   3. after the pass's __syncthreads (which also publishes the ||x||^2 partials) one thread per own row publishes
//      the pair ((A x)_r, A(r,k-1)) with one relaxed store, and every thread forms beta, tau, scale and v exactly as
//      every other CTA does (same data, same summation order => bit-identical v in all CTAs);
//   4. reads every row's pair for its columns.  There is no barrier: a slot of the exchange ring holds a NaN pattern
//      no result can have until its pair arrives, and the reader polls the pair itself.  y = scale (A x) + A(:,k-1)
//      with the owner's fma;
//   5. forms w = tau y - tau^2/2 (y.v) v and the next x = A(0:k-2, k-1) - v w(k-1) - w v(k-1) redundantly.
// Two block-level syncs and one L2 round trip per column; every reduction runs in a fixed order that does not depend
// on the grid, so results are deterministic, identical across CTAs and the same for every grid size; every wait is
// time-limited (device status word, no trap).
//
// What bounds it: latency.  An exchange of 1788 pairs among 148 CTAs alone takes 4700 cycles with an arrival counter
// (store, fence, counter, poll, then the loads) and 2300 with polled pairs; of 412 pairs 3700 and 1900.  Two things make
// the polled form work: neighbouring rows belong to one CTA, so that no two CTAs write one 32-byte sector (with cyclic
// single rows, sectors shared by writers and polled meanwhile, the same exchange took 8000 cycles), and the first poll
// comes only after the Householder scalars, about when the pairs arrive.  Inside the CTA, the rows were bound by
// shared memory (every element loaded and stored each column: 186 KB twice per column and SM at n = 1788); 8 of 14 rows
// in registers leave it 6.  Eight warps instead of sixteen halve the shuffles and the cross-warp sums, and a column's
// code is specialised on the column pairs still active, so that it is straight-line and its dependent chains interleave.
// Whole stage, FP64, before -> after: n = 1788 7.19 -> 4.52 ms (4.0 -> 2.5 us per column), 1203 4.27 -> 2.70,
// 619 1.88 -> 1.21, 412 1.19 -> 0.69; FP32 n = 1788 6.24 -> 3.85 (now, with the last 64 columns in registers and the
// publication's addresses formed ahead: 4.28, 2.52, 1.03, 0.56; FP32 3.56).
//
// The ring has three thirds of H slots; step t uses slot t mod 3H.  In step t = bH + 1, after publishing, the owner
// of a row puts the empty pattern back into its entries of third (b - 1) mod 3 and every thread executes a fence.
// Every CTA has then read all of third (b - 1) mod 3: a CTA reads step s only if it has a row in step s + 1, which it
// publishes after reading, and this CTA has read every pair of step t - 1 = bH.  The third is polled again from step
// (b + 2)H on; by then the reader has seen a later publish of the same owner thread (step bH + 2 or later, H >= 2) and
// executed its own fence of step (b + 1)H + 1, so the emptying happens before the poll.  A fence costs about 1000 cycles
// while stores are in flight, so a third has 32 slots (8: 2 % slower).
#include <type_traits>

#include "common.cuh"
#include "kernels.h"

namespace xtbeig {

namespace {

constexpr int kRowChunk = 8;  // rows whose partial dot products are reduce-scattered together

// Relaxed (morally strong) accesses of the exchange ring: each value of a pair is its own 8- (4-)byte access.
__device__ __forceinline__ void st_pair(double* p, double a, double b) {
  asm volatile("st.relaxed.gpu.global.v2.f64 [%0], {%1, %2};" ::"l"(p), "d"(a), "d"(b) : "memory");
}
__device__ __forceinline__ void ld_pair(const double* p, double& a, double& b) {
  asm volatile("ld.relaxed.gpu.global.v2.f64 {%0, %1}, [%2];" : "=d"(a), "=d"(b) : "l"(p) : "memory");
}
__device__ __forceinline__ void st_pair(float* p, float a, float b) {
  asm volatile("st.relaxed.gpu.global.v2.f32 [%0], {%1, %2};" ::"l"(p), "f"(a), "f"(b) : "memory");
}
__device__ __forceinline__ void ld_pair(const float* p, float& a, float& b) {
  asm volatile("ld.relaxed.gpu.global.v2.f32 {%0, %1}, [%2];" : "=f"(a), "=f"(b) : "l"(p) : "memory");
}

// The empty pattern is all ones (a NaN); a value whose high word is all ones counts as empty, so the publisher turns
// such a NaN (only an input's payload can be one) into the default NaN.
__device__ __forceinline__ bool is_empty(double x) { return __double2hiint(x) == -1; }
__device__ __forceinline__ bool is_empty(float x) { return __float_as_int(x) == -1; }
__device__ __forceinline__ double published(double x) {
  return is_empty(x) ? __longlong_as_double(0x7ff8000000000000ll) : x;
}
__device__ __forceinline__ float published(float x) { return is_empty(x) ? __int_as_float(0x7fc00000) : x; }
template <typename T>
__device__ __forceinline__ T empty_value();
template <>
__device__ __forceinline__ double empty_value<double>() { return __longlong_as_double(-1ll); }
template <>
__device__ __forceinline__ float empty_value<float>() { return __int_as_float(-1); }

template <typename T>
struct __align__(2 * sizeof(T)) Pair {
  T a, b;
};

// A column of the trailing block whose squared norm is below a bound is taken as zero (tau = 0; its elements, but not alpha,
// are dropped).  Where a block vanishes, as in a matrix of low rank, rounding leaves u |A|, u^2 |A|, ... of it column by
// column, until the squares underflow: with a norm good to a few bits v and tau no longer fit together and Q was not
// orthogonal (ones(33): |Q^T Q - I| = 0.13).  The bound is where the sum of n <= 2^14 squares loses its last bits to
// underflow, but never more than 2^-10 u of the largest column so far, so that a matrix that is small itself keeps its
// columns: what is dropped lies below the rounding of the reduction.
template <typename T>
struct ColumnFloor;
template <>
struct ColumnFloor<double> {
  static constexpr double kTiny = 0x1p-1000, kOfLargest = 0x1p-126;
};
template <>
struct ColumnFloor<float> {
  static constexpr float kTiny = 0x1p-110f, kOfLargest = 0x1p-68f;
};
// The bound after a column of squared norm s2.
template <typename T>
__device__ __forceinline__ T next_floor2(T floor2, T s2) {
  return fmax(floor2, fmin(ColumnFloor<T>::kTiny, s2 * ColumnFloor<T>::kOfLargest));
}

// Sum of N values (N a power of two) read from shared memory, as a balanced tree: log2 N dependent additions.
template <int N, typename T>
__device__ __forceinline__ T tree_sum(const T* p, int stride) {
  T v[N];
#pragma unroll
  for (int i = 0; i < N; ++i) v[i] = p[i * stride];
#pragma unroll
  for (int s = 1; s < N; s *= 2)
#pragma unroll
    for (int i = 0; i + s < N; i += 2 * s) v[i] += v[i + s];
  return v[0];
}

// FP64 matrix instruction D = A B (8 x 4 times 4 x 8; lane l holds A[l/4][l%4], B[l%4][l/4] and D[l/4][2(l%4)], + 1).
// With A all ones, D[m][n] is the sum of B's column n, that is of the four lanes of quad n, for every m: a lane receives
// the sums of quads 2(l%4) and 2(l%4) + 1.
__device__ __forceinline__ void quad_sums(double v, double& even, double& odd) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%4, %4};"
               : "=d"(even), "=d"(odd)
               : "d"(1.0), "d"(v), "d"(0.0));
}

// Sum over the warp, in every lane: two matrix instructions (77 cycles) instead of five shuffles (191).
__device__ __forceinline__ double warp_sum_mma(double v) {
  double a, b;
  quad_sums(v, a, b);
  quad_sums(a + b, a, b);
  return a;
}
__device__ __forceinline__ float warp_sum_mma(float v) { return warp_sum(v); }

// The warp-wide sums of ROWS (8 or 4) per-lane values each to out[0 .. ROWS): halves are exchanged (added) across lanes
// 16, 8 and 4, which leaves every row in one quad (in two), whose lanes one matrix instruction sums.  Both forms add in
// the same order, so a row's sum does not depend on how many rows its CTA has.
template <int ROWS>
__device__ __forceinline__ void warp_row_sums(double (&acc)[kRowChunk], double* out) {
  const unsigned lane = threadIdx.x & 31;
  const bool h4 = lane & 16, h3 = lane & 8, h2 = lane & 4;
#pragma unroll
  for (int i = 0; i < ROWS / 2; ++i) {
    const double send = h4 ? acc[i] : acc[i + ROWS / 2], keep = h4 ? acc[i + ROWS / 2] : acc[i];
    acc[i] = keep + __shfl_xor_sync(0xffffffffu, send, 16);
  }
#pragma unroll
  for (int i = 0; i < ROWS / 4; ++i) {
    const double send = h3 ? acc[i] : acc[i + ROWS / 4], keep = h3 ? acc[i + ROWS / 4] : acc[i];
    acc[i] = keep + __shfl_xor_sync(0xffffffffu, send, 8);
  }
  double even, odd;
  if constexpr (ROWS == 8) {
    const double send = h2 ? acc[0] : acc[1], keep = h2 ? acc[1] : acc[0];
    quad_sums(keep + __shfl_xor_sync(0xffffffffu, send, 4), even, odd);
    if (lane < 4) *reinterpret_cast<Pair<double>*>(out + 2 * lane) = Pair<double>{even, odd};
  } else {
    quad_sums(acc[0] + __shfl_xor_sync(0xffffffffu, acc[0], 4), even, odd);
    if (lane < 4) out[lane] = even;  // row l is in quads 2l and 2l + 1
  }
}
template <int ROWS>
__device__ __forceinline__ void warp_row_sums(float (&acc)[kRowChunk], float* out) {
  const unsigned lane = threadIdx.x & 31;
  const bool h4 = lane & 16, h3 = lane & 8, h2 = lane & 4;
#pragma unroll
  for (int i = 0; i < ROWS / 2; ++i) {
    const float send = h4 ? acc[i] : acc[i + ROWS / 2], keep = h4 ? acc[i + ROWS / 2] : acc[i];
    acc[i] = keep + __shfl_xor_sync(0xffffffffu, send, 16);
  }
#pragma unroll
  for (int i = 0; i < ROWS / 4; ++i) {
    const float send = h3 ? acc[i] : acc[i + ROWS / 4], keep = h3 ? acc[i + ROWS / 4] : acc[i];
    acc[i] = keep + __shfl_xor_sync(0xffffffffu, send, 8);
  }
  float r = acc[0];
  if constexpr (ROWS == 8) {
    const float send = h2 ? acc[0] : acc[1], keep = h2 ? acc[1] : acc[0];
    r = keep + __shfl_xor_sync(0xffffffffu, send, 4);
  } else {
    r += __shfl_xor_sync(0xffffffffu, r, 4);
  }
  r += __shfl_xor_sync(0xffffffffu, r, 2);
  r += __shfl_xor_sync(0xffffffffu, r, 1);
  if ((lane & 3) == 0 && (ROWS == 8 || h2 == false)) out[ROWS == 8 ? lane >> 2 : lane >> 3] = r;
}

// One row chunk of the pass over the first JA column pairs: ROWS register rows, or ROWS rows of shared (global) memory,
// whose pairs from FULL on are tested against k (the pairs before lie below k in every thread).  Straight-line code, so that the rows' dependent chains interleave (a
// branch per row and pair left every chain's latency exposed: 5700 cycles instead of 2000 for 13 rows of 1788).
template <int ROWS, int JA, int CPT, typename T>
__device__ __forceinline__ void pass_registers(T (*ra)[CPT], const Pair<T>* vy, T tau, T half, const T* wk, const T* vk,
                                               const T* xs, T* acc) {
  T vr[ROWS], wr[ROWS];
#pragma unroll
  for (int q = 0; q < ROWS; ++q) {
    const Pair<T> o = vy[q];
    vr[q] = -o.a;
    wr[q] = fma(-tau, o.b, half * o.a);  // -w, bit for bit the negative of the owner's w = tau y - half v
  }
#pragma unroll
  for (int i = 0; i < 2 * JA; ++i) {
#pragma unroll
    for (int q = 0; q < ROWS; ++q) {
      T a = fma(vr[q], wk[i], ra[q][i]);
      a = fma(wr[q], vk[i], a);
      ra[q][i] = a;
      acc[q] = fma(a, xs[i], acc[q]);
    }
  }
}

template <int ROWS, int JA, int FULL, int NT, typename T>
__device__ __forceinline__ void pass_memory(T* row0, size_t ldr, int k, const Pair<T>* vy, T tau, T half, const T* wk,
                                            const T* vk, const T* xs, T* acc) {
  // Every load before the first store: the stores could alias the loads for all the compiler knows.
  Pair<T> e[ROWS][JA];
  const int c0 = 2 * (int)threadIdx.x;
  auto in = [&](int j) { return j < FULL || c0 + 2 * j * NT < k; };
#pragma unroll
  for (int q = 0; q < ROWS; ++q)
#pragma unroll
    for (int j = 0; j < JA; ++j) {
      if (j >= FULL) e[q][j] = Pair<T>{T(0), T(0)};
      if (in(j)) e[q][j] = *reinterpret_cast<const Pair<T>*>(row0 + q * ldr + c0 + 2 * j * NT);
    }
  T vr[ROWS], wr[ROWS];
#pragma unroll
  for (int q = 0; q < ROWS; ++q) {
    const Pair<T> o = vy[q];
    vr[q] = -o.a;
    wr[q] = fma(-tau, o.b, half * o.a);
  }
#pragma unroll
  for (int j = 0; j < JA; ++j)
#pragma unroll
    for (int q = 0; q < ROWS; ++q) {
      e[q][j].a = fma(wr[q], vk[2 * j], fma(vr[q], wk[2 * j], e[q][j].a));
      e[q][j].b = fma(wr[q], vk[2 * j + 1], fma(vr[q], wk[2 * j + 1], e[q][j].b));
      acc[q] = fma(e[q][j].b, xs[2 * j + 1], fma(e[q][j].a, xs[2 * j], acc[q]));
    }
#pragma unroll
  for (int q = 0; q < ROWS; ++q)
#pragma unroll
    for (int j = 0; j < JA; ++j)
      if (in(j)) *reinterpret_cast<Pair<T>*>(row0 + q * ldr + c0 + 2 * j * NT) = e[q][j];
}

// kUpperInPlace: the variant that reads the upper triangle of p.afull (== p.aout) in place instead of a full
// symmetric copy, and therefore waits at one grid barrier after loading, before any CTA writes the matrix.
// kSmemRows: rows from RR on are resident in shared memory (known at compile time, so row accesses are shared-memory
// instructions).  CPT columns per thread in pairs; NT CPT >= n.
template <typename T, int NT, int CPT, int RR, bool kUpperInPlace = false, bool kSmemRows = true>
__global__ void __launch_bounds__(NT, 1) sytrd_resident_kernel(SytrdParams<T> p) {
  constexpr int NW = NT / 32, CP = CPT / 2;
  static_assert(RR == 0 || RR == 4 || RR == 8, "register rows: whole, half or none of a reduce-scatter");
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int G = gridDim.x, cta = blockIdx.x, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int n = p.n, R = p.rows_per_cta, H = p.ring_h;
  const size_t ldr = (size_t)p.ldr, slot_ld = sytrd_ring_elems(n, 1) / 3;
  if (ld_volatile_i32(&p.st->code) != 0) return;  // an earlier stage failed: every CTA skips the reduction
  constexpr int BL = sytrd_row_block<T>();
  auto row_of = [&](int q) { return BL * ((q / BL) * G + cta) + (q % BL); };

  // Shared memory (sytrd_smem_bytes): x, (v, y) at own rows, per-warp partial row sums, captured A(r, k-1), block
  // sums, broadcast scalars, rows.
  T* xsm = reinterpret_cast<T*>(smem_raw);                   // [NT * CPT] x of this column
  Pair<T>* vy = reinterpret_cast<Pair<T>*>(xsm + NT * CPT);  // [R + 8] previous (v, y), zero beyond R
  T* red = reinterpret_cast<T*>(vy + R + 8);                 // [NW][R + 8]
  T* colk = red + (size_t)(R + 8) * NW;                      // [8]
  T* bred = colk + 8;                                        // [2][NW]
  T* scal = bred + 2 * NW;                                   // [4], and the column floor before an even and an odd column
  T* rows = nullptr;
  if constexpr (kSmemRows) {
    const size_t off = (size_t)(reinterpret_cast<unsigned char*>(scal + 6) - smem_raw);
    rows = reinterpret_cast<T*>(smem_raw + ((off + 15) & ~size_t(15)));
  } else {
    rows = p.grows + (size_t)cta * R * ldr;
  }

  // Load own rows (row r of the symmetric matrix is its column r: contiguous).
  T ra[RR > 0 ? RR : 1][CPT];
  auto load = [&](int r, int c) -> T {
    if constexpr (kUpperInPlace)
      return c <= r ? p.afull[c + (size_t)r * p.ldf] : p.afull[r + (size_t)c * p.ldf];
    else
      return p.afull[c + (size_t)r * p.ldf];
  };
#pragma unroll
  for (int q = 0; q < RR; ++q) {
    const int r = row_of(q);
#pragma unroll
    for (int i = 0; i < CPT; ++i) {
      const int c = 2 * (tid + (i >> 1) * NT) + (i & 1);
      ra[q][i] = (r < n && c < n) ? load(r, c) : T(0);
    }
  }
  for (int q = RR; q < R; ++q) {
    const int r = row_of(q);
    if (r >= n) break;
    T* dst = rows + (size_t)(q - RR) * ldr;
    for (int c = tid; c < (int)ldr; c += NT) dst[c] = c < n ? load(r, c) : T(0);
  }

  T xs[CPT], vk[CPT], wk[CPT];
#pragma unroll
  for (int i = 0; i < CPT; ++i) {
    const int c = 2 * (tid + (i >> 1) * NT) + (i & 1);
    const T x = (n >= 1 && c < n - 1) ? load(n - 1, c) : T(0);
    xsm[c] = x;
    if (c == n - 2) scal[0] = x;
    xs[i] = c < n - 2 ? x : T(0);
    vk[i] = wk[i] = T(0);
  }
  for (int q = tid; q < R + 8; q += NT) vy[q] = Pair<T>{T(0), T(0)};
  if (tid < 2) scal[4 + tid] = T(0);
  if (cta == 0 && tid == 0 && n >= 1) {
    T dn = load(n - 1, n - 1);
    p.d[n - 1] = dn;
    p.aout[(size_t)(n - 1) + (size_t)(n - 1) * p.lda] = dn;
  }
  __syncthreads();
  if constexpr (kUpperInPlace) {
    unsigned epoch = 0;
    if (!group_barrier(p.counter, (unsigned)G, epoch, p.st, p.limit_ns)) return;
  }

  // tau and tau^2/2 (y.v) of the previous step: with the previous step's (v, y) at own rows they give its w at own
  // rows, w = tau y - half v, exactly as the owner of each column forms w.
  T tau_prev = T(0), half_prev = T(0);
  bool dead = false;  // a wait ran out or another CTA failed: this thread polls no more (the status word is set)
  int phase = 0, third = 2;  // step index mod H; third emptied at phase 1
  bool first_block = true;
  const int k_end = p.k_stop > 0 ? p.k_stop + 1 : 1;  // last step this kernel runs
  int nq = 0;                                          // own rows r < k (ascending, so they retire from the end)
  while (nq < R && row_of(nq) < n - 1) ++nq;
  int last_row = nq > 0 ? row_of(nq - 1) : -1;
  const int first_row = row_of(0);
  if (first_row >= n - 1 && cta > 0) return;  // no row in any step
  int ja = (n - 1 + 2 * NT - 1) / (2 * NT);  // column pairs per thread that reach below k
  T* xch = p.xch;                            // ((A x)_r, A(r, k-1)) pairs of this step
  // Thread q publishes own row q (rows beyond the block's threads: a loop): where it finds the row's sums and its
  // A(r, k-1), formed once, since the publication is on every CTA's critical path.
  const int my_row = row_of(tid);
  const T* my_sums = red + min(tid, R);
  const T* my_col = tid < RR || tid >= R ? colk + min(tid, 7) : rows + (size_t)(tid - RR) * ldr;
  const int my_step = tid < RR ? 0 : 1;
  T* const ring_end = p.xch + (size_t)3 * H * slot_ld;
  for (int k = n - 1; k >= k_end; --k) {
    if (last_row >= k) {
      --nq;
      last_row = nq > 0 ? row_of(nq - 1) : -1;
    }
    if (2 * NT * (ja - 1) >= k) --ja;

    // One column, over the first JA column pairs of every thread (the others lie beyond k).
    // FULL pairs lie wholly below k: all but the last, unless this code serves several counts of active pairs (CP 8: 1 to
    // 4, and 5 to 8), where a pair past the active ones would lie in the next row.
    auto step = [&](auto JA) {
      constexpr int J = decltype(JA)::value, E = 2 * J, FULL = CP <= 4 ? J - 1 : 0;
      // ||x||^2 of x = A(0:k-2, k): per-warp partials, summed after the pass's __syncthreads.
      T part;
      {
        T s0 = T(0), s1 = T(0);
#pragma unroll
        for (int i = 0; i < E; i += 2) {
          s0 = fma(xs[i], xs[i], s0);
          s1 = fma(xs[i + 1], xs[i + 1], s1);
        }
        part = warp_sum_mma(s0 + s1);
      }
      // ---- 1 + 2. fused pass: previous rank-2 update + A x over own rows r < k.  Register rows beyond nq and columns
      //      from k on need no test: v, w and x are zero there, and no one reads the sums.
      if constexpr (RR > 0) {
        T acc[kRowChunk];
#pragma unroll
        for (int q = 0; q < kRowChunk; ++q) acc[q] = T(0);
        if constexpr (RR == 8) {
          if (nq > 4) pass_registers<8, J, CPT, T>(ra, vy, tau_prev, half_prev, wk, vk, xs, acc);
          else if (nq > 2) pass_registers<4, J, CPT, T>(ra, vy, tau_prev, half_prev, wk, vk, xs, acc);
          else pass_registers<2, J, CPT, T>(ra, vy, tau_prev, half_prev, wk, vk, xs, acc);
          warp_row_sums<8>(acc, red + warp * (R + 8));
        } else {
          if (nq > 2) pass_registers<4, J, CPT, T>(ra, vy, tau_prev, half_prev, wk, vk, xs, acc);
          else pass_registers<2, J, CPT, T>(ra, vy, tau_prev, half_prev, wk, vk, xs, acc);
          warp_row_sums<4>(acc, red + warp * (R + 8));
        }
      }
      for (int q0 = RR; q0 < nq; q0 += kRowChunk) {
        T acc[kRowChunk];
#pragma unroll
        for (int q = 0; q < kRowChunk; ++q) acc[q] = T(0);
        const int rem = nq - q0;
        T* row = rows + (size_t)(q0 - RR) * ldr;
        const Pair<T>* o = vy + q0;
        // Rows in pairs, so at most one row beyond nq (its storage exists: R is even); sums beyond nq are not read.  Beside
        // more than eight columns' x, v and w the registers hold one column pair of two rows: all eight pairs at once
        // (n > 8192, FP64) spilled: n = 9500 2.02 s, 13000 5.64 s; one at a time 1.57 and 3.65.
        auto pair = [&](int i) {
          if constexpr (J <= 4) {
            pass_memory<2, J, FULL, NT, T>(row + i * ldr, ldr, k, o + i, tau_prev, half_prev, wk, vk, xs, acc + i);
          } else {
#pragma unroll
            for (int j = 0; j < J; ++j)
              pass_memory<2, 1, 0, NT, T>(row + i * ldr + 2 * j * NT, ldr, k - 2 * j * NT, o + i, tau_prev, half_prev,
                                          wk + 2 * j, vk + 2 * j, xs + 2 * j, acc + i);
          }
        };
        pair(0);
        if (rem > 2) pair(2);
        if (rem > 4) {
          pair(4);
          if (rem > 6) pair(6);
          warp_row_sums<8>(acc, red + warp * (R + 8) + q0);
        } else {
          warp_row_sums<4>(acc, red + warp * (R + 8) + q0);
        }
      }
      // A(r, k-1) of the register rows, from the thread that holds column k-1 (the others are read from the row).
      if constexpr (RR > 0) {
#pragma unroll
        for (int j = 0; j < J; ++j) {
          if (tid + j * NT == (k - 1) >> 1) {
#pragma unroll
            for (int q = 0; q < RR; ++q) colk[q] = ((k - 1) & 1) ? ra[q][2 * j + 1] : ra[q][2 * j];
          }
        }
      }
      if (lane == 0) bred[warp] = part;
      __syncthreads();  // publishes red, colk, the rows, the ||x||^2 partials and alpha
      // ---- 3. publish ((A x)_r, A(r,k-1)) for own rows, one thread per row; neighbouring rows fill a 32-byte sector in
      //      one store.  The consumer forms y_r = scale (A x)_r + A(r, k-1) with the same fma as the owner.
      T ax_own = T(0), col_own = T(0);
      if (tid < nq) {
        ax_own = tree_sum<NW>(my_sums, R + 8);
        col_own = my_col[my_step * (k - 1)];
        st_pair(xch + 2 * (size_t)my_row, published(ax_own), published(col_own));
      }
      for (int q = tid + NT; q < nq; q += NT) {
        const T ax = tree_sum<NW>(red + q, R + 8);
        st_pair(xch + 2 * (size_t)row_of(q), published(ax), published(rows[(size_t)(q - RR) * ldr + (k - 1)]));
        red[q] = ax;
      }
      // ---- 4. Householder vector (identical in every CTA: same data, same order).
      const T xn2 = tree_sum<NW>(bred, 1);
      const T alpha = scal[0], s2 = alpha * alpha + xn2, floor2 = scal[4 + (k & 1)];
      T beta, tau, scale;
      if (xn2 == T(0) || s2 < floor2) {
        beta = alpha; tau = T(0); scale = T(0);
      } else {
        // beta = -sign(alpha) ||(alpha, x)||, tau = (beta - alpha)/beta = 1 + |alpha|/||.||: one reciprocal square
        // root and one division.
        const T rn = rsqrt(s2);
        const T nrm = s2 * rn;
        beta = alpha >= T(0) ? -nrm : nrm;
        tau = T(1) + fabs(alpha) * rn;
        scale = T(1) / (alpha - beta);
      }
#pragma unroll
      for (int i = 0; i < E; ++i) {
        const int c = 2 * (tid + (i >> 1) * NT) + (i & 1);
        vk[i] = c == k - 1 ? T(1) : xs[i] * scale;  // zero from k on
      }
      // ---- 5. read every row's pair for this thread's columns, polling the pairs themselves.
      T y[E], col[E];
#pragma unroll
      for (int i = 0; i < E; ++i) {
        const int c = 2 * (tid + (i >> 1) * NT) + (i & 1);
        y[i] = col[i] = T(0);
        if (c < k) ld_pair(xch + 2 * c, y[i], col[i]);
      }
      // In the shadow of the loads: own rows' (v, y) and output entries, the scalars, the ring's upkeep.
      auto keep_row = [&](int q, int r, T ax, T ck) {
        const T v = r < k - 1 ? xsm[r] * scale : T(1);
        vy[q] = Pair<T>{v, fma(scale, ax, ck)};
        p.aout[r + (size_t)k * p.lda] = r < k - 1 ? v : beta;
      };
      if (tid < nq) keep_row(tid, my_row, ax_own, col_own);
      for (int q = tid + NT; q < nq; q += NT) keep_row(q, row_of(q), red[q], rows[(size_t)(q - RR) * ldr + (k - 1)]);
      if (tid == NT - 1) {
        scal[4 + ((k - 1) & 1)] = next_floor2(floor2, s2);
        if (cta == 0) { p.e[k - 1] = beta; p.tau[k - 1] = tau; }
      }
      if (phase == 1) {  // empty the third that every CTA has finished reading (see above)
        if (!first_block) {
          T* base = p.xch + (size_t)third * H * slot_ld;
          for (int q = tid; q < R; q += NT)
            if (row_of(q) < n)
              for (int s = 0; s < H; ++s)
                st_pair(base + (size_t)s * slot_ld + 2 * row_of(q), empty_value<T>(), empty_value<T>());
        }
        __threadfence();
      }
      // A CTA without a row in the next step is done: it must not read this step's pairs, because nothing would tell
      // the others when it has finished, and they empty the slot some steps later.  (Row 0's CTA stays to the end, and
      // the last step's pairs are not emptied.)
      if (first_row >= k - 1 && k > k_end) return false;
      {
        uint64_t t0 = 0;
        unsigned spins = 0;
        while (!dead) {
          bool waiting = false;
#pragma unroll
          for (int i = 0; i < E; ++i) waiting = waiting || is_empty(y[i]) || is_empty(col[i]);
          if (p.extra_members && tid == 0) {  // failure-detection hook: a pair that is never published
            T ea, eb;
            ld_pair(xch + 2 * (size_t)n, ea, eb);
            waiting = waiting || is_empty(ea);
          }
          if (!waiting) break;
#pragma unroll
          for (int i = 0; i < E; ++i) {
            const int c = 2 * (tid + (i >> 1) * NT) + (i & 1);
            if (is_empty(y[i]) || is_empty(col[i])) ld_pair(xch + 2 * c, y[i], col[i]);
          }
          if ((++spins & 63u) == 0) {
            if (ld_volatile_i32(&p.st->code) != 0) dead = true;
            const uint64_t now = global_ns();
            if (t0 == 0) t0 = now;
            else if (now - t0 > p.limit_ns) {
              set_status(p.st, kStatusBarrierTimeout, 0, n - k);
              dead = true;
            }
          }
        }
      }
      __syncwarp();
      // y(k-1) and A(k-1,k-1) for w(k-1) and d(k-1), published through the same __syncthreads as y.v.
      {
        T s0 = T(0), s1 = T(0);
#pragma unroll
        for (int i = 0; i < E; ++i) {
          const int c = 2 * (tid + (i >> 1) * NT) + (i & 1);
          y[i] = fma(scale, y[i], col[i]);
          if (c == k - 1) { scal[1] = y[i]; scal[2] = col[i]; }
          if (i & 1) s1 = fma(y[i], vk[i], s1);
          else s0 = fma(y[i], vk[i], s0);
        }
        const T pyv = warp_sum_mma(s0 + s1);
        if (lane == 0) bred[NW + warp] = pyv;
      }
      __syncthreads();
      const T yv = tree_sum<NW>(bred + NW, 1);
      const T half = T(0.5) * tau * tau * yv;
      const T wkm1 = tau * scal[1] - half;  // v(k-1) = 1
      if (cta == 0 && tid == NT - 1) {
        const T dk = scal[2] - T(2) * wkm1;  // A(k-1,k-1) after this step's update
        p.d[k - 1] = dk;
        p.aout[(size_t)(k - 1) + (size_t)(k - 1) * p.lda] = dk;
      }
#pragma unroll
      for (int j = 0; j < J; ++j) {
        const int c0 = 2 * (tid + j * NT);
        Pair<T> xp;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const int i = 2 * j + h, c = c0 + h;
          const T w = fma(tau, y[i], -(half * vk[i]));
          const T x = c < k - 1 ? col[i] - vk[i] * wkm1 - w : T(0);
          if (c == k - 2) scal[0] = x;
          xs[i] = c < k - 2 ? x : T(0);
          wk[i] = w;
          (h ? xp.b : xp.a) = x;
        }
        *reinterpret_cast<Pair<T>*>(xsm + c0) = xp;
      }
      tau_prev = tau;
      half_prev = half;
      return true;
    };
    bool more;
    if constexpr (CP == 1) {
      more = step(std::integral_constant<int, 1>{});
    } else if constexpr (CP == 2) {
      if (ja == 2) more = step(std::integral_constant<int, 2>{});
      else more = step(std::integral_constant<int, 1>{});
    } else if constexpr (CP == 4) {
      if (ja == 4) more = step(std::integral_constant<int, 4>{});
      else if (ja == 3) more = step(std::integral_constant<int, 3>{});
      else if (ja == 2) more = step(std::integral_constant<int, 2>{});
      else more = step(std::integral_constant<int, 1>{});
    } else {
      if (ja > 4) more = step(std::integral_constant<int, CP>{});
      else more = step(std::integral_constant<int, 4>{});
    }
    if (!more) return;
    xch += slot_ld;
    if (xch == ring_end) xch = p.xch;
    if (++phase == H) {
      phase = 0;
      first_block = false;
      third = third == 2 ? 0 : third + 1;
    }
  }
  // Hand-over: the pending update of step k_stop + 1 applied to the trailing block, whose full symmetric rows go to
  // `hand` (row r of the block is its column r).  vy and the scalars are this CTA's own; vk and wk were formed after
  // the last exchange, so every row of the block is complete.
  if (p.k_stop > 0 && k_end <= n - 1) {
    const int m = p.k_stop + 1;
    if (cta == 0 && tid == 0) *p.floor2 = scal[4 + ((k_end - 1) & 1)];
    auto hand_row = [&](int q, auto get) {
      const int r = row_of(q);
      const Pair<T> o = vy[q];
      const T vr = o.a, wr = fma(tau_prev, o.b, -(half_prev * vr));
      T* dst = p.hand + (size_t)r * p.ldh;
#pragma unroll
      for (int i = 0; i < CPT; ++i) {
        const int c = 2 * (tid + (i >> 1) * NT) + (i & 1);
        if (c < m) dst[c] = fma(-wr, vk[i], fma(-vr, wk[i], get(i, c)));
      }
    };
#pragma unroll
    for (int q = 0; q < RR; ++q)
      if (row_of(q) < m) hand_row(q, [&](int i, int) { return ra[q][i]; });
    for (int q = RR; q < R && row_of(q) < m; ++q)
      hand_row(q, [&](int, int c) { return rows[(size_t)(q - RR) * ldr + c]; });
  }
}

// Reduce-scatter of ROWS (16, 8 or 4) per-lane values per warp: the warp-wide sum of row i to out[i * stride].  Halves
// are exchanged across lanes 16, 8, 4 as in warp_row_sums; one matrix instruction then sums the quads of each value
// that is left (16 rows leave two per lane).
template <int ROWS>
__device__ __forceinline__ void warp_row_sums_strided(double (&acc)[ROWS], double* out, int stride) {
  const unsigned lane = threadIdx.x & 31;
  int rows = ROWS;
#pragma unroll
  for (int bit = 16; bit >= 4; bit /= 2) {
    const bool hi = lane & bit;
    if (rows > 1) {
#pragma unroll
      for (int i = 0; i < ROWS / 2; ++i) {
        if (i < rows / 2) {
          const double send = hi ? acc[i] : acc[i + rows / 2], keep = hi ? acc[i + rows / 2] : acc[i];
          acc[i] = keep + __shfl_xor_sync(0xffffffffu, send, bit);
        }
      }
      rows /= 2;
    } else {
      acc[0] += __shfl_xor_sync(0xffffffffu, acc[0], bit);
    }
  }
  // Quad n (lanes 4n .. 4n + 3) now holds rows n ROWS/8 + s (ROWS 4: row n / 2).
  constexpr int S = ROWS >= 8 ? ROWS / 8 : 1;
#pragma unroll
  for (int s = 0; s < S; ++s) {
    double even, odd;
    quad_sums(acc[s], even, odd);
    if (lane < 4) {
      if constexpr (ROWS == 4) {
        out[lane * stride] = even;
      } else {
        out[(2 * lane * S + s) * stride] = even;
        out[((2 * lane + 1) * S + s) * stride] = odd;
      }
    }
  }
}
template <int ROWS>
__device__ __forceinline__ void warp_row_sums_strided(float (&acc)[ROWS], float* out, int stride) {
  const unsigned lane = threadIdx.x & 31;
#pragma unroll
  for (int i = 0; i < ROWS; ++i) {
    const float r = warp_sum(acc[i]);
    if (lane == (unsigned)i) out[i * stride] = r;
  }
}

// The last columns on one CTA, the trailing block (order m <= M) in registers: warp w of M / 16 owns rows w, w + NW, ...
// (16 of them), lane l the columns l, l + 32, ...  Per column k, as in the grid kernel: the pass applies the previous
// rank-2 update and sums A x at the warp's rows; one block sync exchanges (A x)_r and A(r, k-1) through shared memory
// (two alternating buffers); every warp then forms y, v, w and the next x itself, from the same data in the same order,
// so no other sync is needed.  For M = 64 one more warp owns no rows: it forms the Householder scalars of the same x while
// the others pass over their rows (a dependent chain of a sum, a reciprocal square root and a division).
// A warp's own copy of (v, w) in shared memory gives it the values at its rows.  Bound by latency: the pass and its
// reduce-scatter, one sync, a warp sum by matrix instruction.  It replaced a kernel that kept the block in shared memory
// with four block syncs and two shuffled sums per column (2.0 us per column of a block of 64, now 0.6: 130 -> 40 us).
template <typename T, int M>
__global__ void __launch_bounds__(2 * M + (M == 64 ? 32 : 0), 1) sytrd_tail_kernel(SytrdParams<T> p, int skip_dinit) {
  constexpr int NW = M / 16, CJ = M / 32;
  constexpr bool kScalarWarp = M == 64;  // M = 128: the registers of a ninth warp would make the others spill
  __shared__ Pair<T> vw[NW][M];  // each warp's (v, w)
  __shared__ T ax_s[2][M], col_s[2][M], scal_s[2][4];
  const int m = p.n, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  if (ld_volatile_i32(&p.st->code) != 0) return;  // an earlier stage failed
  T a[16][CJ], x[CJ], v[CJ], w[CJ];
#pragma unroll
  for (int i = 0; i < 16; ++i) {
    const int r = warp + NW * i;
#pragma unroll
    for (int j = 0; j < CJ; ++j) {
      const int c = lane + 32 * j;
      a[i][j] = (warp < NW && r < m && c < m) ? p.afull[(size_t)r * p.ldf + c] : T(0);
    }
  }
#pragma unroll
  for (int j = 0; j < CJ; ++j) {
    const int c = lane + 32 * j;
    x[j] = (m >= 2 && c < m - 1) ? p.afull[(size_t)(m - 1) * p.ldf + c] : T(0);
    v[j] = w[j] = T(0);
    if (warp < NW) vw[warp][c] = Pair<T>{T(0), T(0)};
  }
  if (!skip_dinit && tid == 0 && m >= 1) {
    const T dn = p.afull[(size_t)(m - 1) * p.ldf + (m - 1)];
    p.d[m - 1] = dn;
    p.aout[(size_t)(m - 1) + (size_t)(m - 1) * p.lda] = dn;
  }
  T floor2 = skip_dinit ? *p.floor2 : T(0);
  __syncwarp();
  for (int k = m - 1; k >= 1; --k) {
    // One column over the first J column groups and ROWS rows per warp (the others lie beyond k).
    auto step = [&](auto Jc, auto Rc) {
      constexpr int J = decltype(Jc)::value, ROWS = decltype(Rc)::value;
      const int buf = k & 1, lk = (k - 1) & 31, jk = (k - 1) >> 5;
      T xs[J];
#pragma unroll
      for (int j = 0; j < J; ++j) xs[j] = lane + 32 * j < k - 1 ? x[j] : T(0);
      // ||x(0:k-2)||^2, alpha = x(k-1) and the Householder scalars.
      T beta, tau, scale;
      auto scalars = [&]() {
        T part = T(0), alpha = T(0);
#pragma unroll
        for (int j = 0; j < J; ++j) {
          part = fma(xs[j], xs[j], part);
          if (j == jk) alpha = __shfl_sync(0xffffffffu, x[j], lk);
        }
        const T xn2 = warp_sum_mma(part), s2 = alpha * alpha + xn2;
        const bool none = xn2 == T(0) || s2 < floor2;
        floor2 = next_floor2(floor2, s2);
        if (none) {
          beta = alpha; tau = T(0); scale = T(0);
        } else {
          const T rn = rsqrt(s2);
          const T nrm = s2 * rn;
          beta = alpha >= T(0) ? -nrm : nrm;
          tau = T(1) + fabs(alpha) * rn;
          scale = T(1) / (alpha - beta);
        }
      };
      if (warp < NW) {
        // Previous rank-2 update and A x at own rows (v = w = x = 0 beyond the block).
        T acc[ROWS];
#pragma unroll
        for (int i = 0; i < ROWS; ++i) {
          const Pair<T> o = vw[warp][warp + NW * i];
          acc[i] = T(0);
#pragma unroll
          for (int j = 0; j < J; ++j) {
            T e = fma(-o.a, w[j], a[i][j]);
            e = fma(-o.b, v[j], e);
            a[i][j] = e;
            acc[i] = fma(e, xs[j], acc[i]);
          }
        }
        // A(r, k-1) of own rows, from the lane that holds column k-1.
#pragma unroll
        for (int j = 0; j < J; ++j) {
          if (j == jk) {
#pragma unroll
            for (int i = 0; i < ROWS; ++i)
              if (lane == lk) col_s[buf][warp + NW * i] = a[i][j];
          }
        }
        warp_row_sums_strided<ROWS>(acc, &ax_s[buf][warp], NW);
      } else {
        scalars();
        if (lane == 0) {
          scal_s[buf][0] = tau;
          scal_s[buf][1] = scale;
          scal_s[buf][2] = beta;
        }
      }
      if constexpr (!kScalarWarp) scalars();
      __syncthreads();
      if constexpr (kScalarWarp) {
        tau = scal_s[buf][0];
        scale = scal_s[buf][1];
        beta = scal_s[buf][2];
      }
      T y[J], col[J], pyv = T(0), yk = T(0), ck = T(0);
#pragma unroll
      for (int j = 0; j < J; ++j) {
        const int c = lane + 32 * j;
        const bool in = c < k;
        col[j] = in ? col_s[buf][c] : T(0);
        y[j] = in ? fma(scale, ax_s[buf][c], col[j]) : T(0);
        v[j] = c == k - 1 ? T(1) : xs[j] * scale;
        pyv = fma(y[j], v[j], pyv);
        if (j == jk) {
          yk = __shfl_sync(0xffffffffu, y[j], lk);
          ck = col[j];
        }
      }
      const T half = T(0.5) * tau * tau * warp_sum_mma(pyv);
      const T wkm1 = tau * yk - half;  // v(k-1) = 1
#pragma unroll
      for (int j = 0; j < J; ++j) {
        const int c = lane + 32 * j;
        w[j] = fma(tau, y[j], -(half * v[j]));
        x[j] = c < k - 1 ? col[j] - v[j] * wkm1 - w[j] : T(0);
        if (warp < NW) vw[warp][c] = Pair<T>{v[j], w[j]};
      }
      __syncwarp();
      if (warp == (kScalarWarp ? NW : k % NW)) {  // the output column
#pragma unroll
        for (int j = 0; j < J; ++j) {
          const int c = lane + 32 * j;
          if (c < k) p.aout[(size_t)c + (size_t)k * p.lda] = c < k - 1 ? v[j] : beta;
        }
        if (lane == lk) {
          const T dk = ck - T(2) * wkm1;  // A(k-1,k-1) after this step's update
          p.e[k - 1] = beta;
          p.tau[k - 1] = tau;
          p.d[k - 1] = dk;
          p.aout[(size_t)(k - 1) + (size_t)(k - 1) * p.lda] = dk;
        }
      }
    };
    using std::integral_constant;
    if constexpr (CJ == 4) {
      if (k > 96) step(integral_constant<int, 4>{}, integral_constant<int, 16>{});
      else if (k > 64) step(integral_constant<int, 3>{}, integral_constant<int, 16>{});
      else if (k > 32) step(integral_constant<int, 2>{}, integral_constant<int, 8>{});
      else step(integral_constant<int, 1>{}, integral_constant<int, 4>{});
    } else {
      if (k > 32) step(integral_constant<int, 2>{}, integral_constant<int, 16>{});
      else step(integral_constant<int, 1>{}, integral_constant<int, 8>{});
    }
  }
}

template <typename T, int NT, int CPT, int RR>
cudaError_t launch_one(const SytrdParams<T>& p, int G, size_t smem, cudaStream_t s) {
  auto kern = p.use_smem ? sytrd_resident_kernel<T, NT, CPT, RR, false, true>
                         : sytrd_resident_kernel<T, NT, CPT, RR, false, false>;
  cudaError_t err = allow_max_dynamic_smem(kern);
  if (err != cudaSuccess) return err;
  void* args[] = {(void*)&p};
  err = cudaLaunchCooperativeKernel((void*)kern, dim3(G), dim3(NT), args, smem, s);
  note_launches();
  return err;
}

// The in-place kernel of a plan, or null: every plan of n <= 2048, whose rows per CTA depend on the device's SMs.
using UpperKernel = void (*)(SytrdParams<double>);
UpperKernel upper_inplace_kernel(const SytrdPlan& pl) {
  switch (pl.threads * 1000 + pl.cpt * 10 + pl.reg_rows) {
    case 128024: return sytrd_resident_kernel<double, 128, 2, 4, true>;
    case 128028: return sytrd_resident_kernel<double, 128, 2, 8, true>;
    case 128044: return sytrd_resident_kernel<double, 128, 4, 4, true>;
    case 128048: return sytrd_resident_kernel<double, 128, 4, 8, true>;
    case 256044: return sytrd_resident_kernel<double, 256, 4, 4, true>;
    case 256048: return sytrd_resident_kernel<double, 256, 4, 8, true>;
    case 256088: return sytrd_resident_kernel<double, 256, 8, 8, true>;
  }
  return nullptr;
}

// Every slot of the ring starts empty (all ones), as far as the launch uses it.
template <typename T>
cudaError_t empty_ring(const SytrdParams<T>& p, cudaStream_t s) {
  return cudaMemsetAsync(p.xch, 0xff, sytrd_ring_elems(p.n, p.ring_h) * sizeof(T), s);
}

}  // namespace

// The in-place variant (upper triangle read where it lies; rows on chip; FP64; n <= 2048).
bool sytrd_upper_inplace_supported(const SytrdPlan& pl) { return pl.rows_in_smem && upper_inplace_kernel(pl) != nullptr; }

cudaError_t sytrd_launch_upper_inplace(const SytrdParams<double>& p, const SytrdPlan& pl, cudaStream_t s) {
  if (p.n <= 0) return cudaSuccess;
  if (!sytrd_upper_inplace_supported(pl)) return cudaErrorInvalidValue;
  cudaError_t err = empty_ring(p, s);
  if (err != cudaSuccess) return err;
  const UpperKernel kern = upper_inplace_kernel(pl);
  err = allow_max_dynamic_smem(kern);
  if (err != cudaSuccess) return err;
  void* args[] = {(void*)&p};
  err = cudaLaunchCooperativeKernel((void*)kern, dim3(pl.grid), dim3(pl.threads), args, pl.smem, s);
  note_launches();
  return err;
}

template <typename T>
size_t sytrd_smem_bytes(int n, int R, int NT, int cpt, int smem_rows, int* ldr_out) {
  const int align = 16 / (int)sizeof(T);
  const int ldr = ((n + align - 1) / align) * align;
  const int NW = NT / 32;
  const size_t elems = (size_t)NT * cpt + 2 * ((size_t)R + 8) + ((size_t)R + 8) * NW + 8 + 2 * (size_t)NW + 6;
  size_t bytes = (elems * sizeof(T) + 15) & ~size_t(15);
  bytes += (size_t)smem_rows * ldr * sizeof(T);
  if (ldr_out) *ldr_out = ldr;
  return bytes;
}

template <typename T>
SytrdPlan sytrd_plan(int n, int num_sms, size_t max_smem, int grid_override) {
  SytrdPlan pl{};
  // Small problems: fewer CTAs, at least ~4 rows each.
  pl.grid = grid_override > 0 ? grid_override : max(1, min(num_sms, (n + 3) / 4));
  // Few warps keep the block syncs and cross-warp sums short; at least four, one per scheduler.
  if (n <= 256) { pl.threads = 128; pl.cpt = 2; }
  else if (n <= 512) { pl.threads = 128; pl.cpt = 4; }
  else if (n <= 1024) { pl.threads = 256; pl.cpt = 4; }
  else if (n <= 2048) { pl.threads = 256; pl.cpt = 8; }
  else if (n <= 4096) { pl.threads = 512; pl.cpt = 8; }
  else { pl.threads = 1024; pl.cpt = n <= 8192 ? 8 : 16; }
  // Registers hold the rows of a CTA that has few of them; blocks of more than 256 threads have none to spare.
  constexpr int BL = sytrd_row_block<T>();
  // A chosen grid so small that even the sums of a CTA's rows outgrow its shared memory is raised to one that works: the
  // results are the same for every grid.
  for (;; ++pl.grid) {
    pl.rows_per_cta = BL * (((n + BL - 1) / BL + pl.grid - 1) / pl.grid);
    if (pl.grid >= num_sms || sytrd_smem_bytes<T>(n, pl.rows_per_cta, pl.threads, pl.cpt, 0, nullptr) <= max_smem) break;
  }
  const int reg_rows = pl.reg_rows = pl.threads > 256 ? 0 : pl.rows_per_cta <= 4 ? 4 : 8;
  const int others = max(0, pl.rows_per_cta - reg_rows);
  const size_t with_rows = sytrd_smem_bytes<T>(n, pl.rows_per_cta, pl.threads, pl.cpt, others, &pl.ldr);
  pl.rows_in_smem = with_rows <= max_smem;
  pl.smem = pl.rows_in_smem ? with_rows : sytrd_smem_bytes<T>(n, pl.rows_per_cta, pl.threads, pl.cpt, 0, nullptr);
  pl.supported = (size_t)pl.threads * pl.cpt >= (size_t)n && pl.cpt <= 16;
  return pl;
}

template <typename T>
cudaError_t sytrd_launch(const SytrdParams<T>& p, const SytrdPlan& pl, cudaStream_t s) {
  if (p.n <= 0) return cudaSuccess;
  const cudaError_t err = empty_ring(p, s);
  if (err != cudaSuccess) return err;
  switch (pl.threads * 1000 + pl.cpt * 10 + pl.reg_rows) {
    case 128024: return launch_one<T, 128, 2, 4>(p, pl.grid, pl.smem, s);
    case 128028: return launch_one<T, 128, 2, 8>(p, pl.grid, pl.smem, s);
    case 128044: return launch_one<T, 128, 4, 4>(p, pl.grid, pl.smem, s);
    case 128048: return launch_one<T, 128, 4, 8>(p, pl.grid, pl.smem, s);
    case 256044: return launch_one<T, 256, 4, 4>(p, pl.grid, pl.smem, s);
    case 256048: return launch_one<T, 256, 4, 8>(p, pl.grid, pl.smem, s);
    case 256088: return launch_one<T, 256, 8, 8>(p, pl.grid, pl.smem, s);
    case 512080: return launch_one<T, 512, 8, 0>(p, pl.grid, pl.smem, s);
    case 1024080: return launch_one<T, 1024, 8, 0>(p, pl.grid, pl.smem, s);
    case 1024160: return launch_one<T, 1024, 16, 0>(p, pl.grid, pl.smem, s);
  }
  return cudaErrorInvalidValue;
}

template <typename T>
cudaError_t sytrd_tail_launch(const SytrdParams<T>& p, int skip_dinit, cudaStream_t s) {
  if (p.n <= 0) return cudaSuccess;
  if (p.n > kSytrdTailMax) return cudaErrorInvalidValue;
  if (p.n <= 64) sytrd_tail_kernel<T, 64><<<1, 160, 0, s>>>(p, skip_dinit);
  else sytrd_tail_kernel<T, 128><<<1, 256, 0, s>>>(p, skip_dinit);
  note_launches();
  return cudaGetLastError();
}

template cudaError_t sytrd_tail_launch<double>(const SytrdParams<double>&, int, cudaStream_t);
template cudaError_t sytrd_tail_launch<float>(const SytrdParams<float>&, int, cudaStream_t);
template SytrdPlan sytrd_plan<double>(int, int, size_t, int);
template SytrdPlan sytrd_plan<float>(int, int, size_t, int);
template cudaError_t sytrd_launch<double>(const SytrdParams<double>&, const SytrdPlan&, cudaStream_t);
template cudaError_t sytrd_launch<float>(const SytrdParams<float>&, const SytrdPlan&, cudaStream_t);

}  // namespace xtbeig
