// Cholesky factor S = U^T U and its explicit inverse X = U^-1 for the generalized problem H C = S C e.
//
// xTB factors S once per geometry (mctc_potrf) and reduces every cycle with dsygst or with the congruence
// H' = X^T H X, X = U^-1 (xtb #1466; reference scripts/kernels/congruence.c:1-52 studies it; EigenBench's dump reader
// does dpotrf, dtrtri and two dtrmm: Sources/EigenBench/main.swift:167-172).
//
// B200 design: ONE persistent cooperative kernel produces both factors (a chain of ~160 small kernels spent most of
// its time in launch and pipeline-fill latency).  Blocks of 64 columns, right-looking, with grid barriers:
//   step j:  B  all CTAs: block row U(j, j+1:) = X(j,j)^T A(j, j+1:)       (64 x 64 DMMA tiles, in place)
//            --- barrier ---
//            C  CTA 0: tile (j+1, j+1) of the trailing update, then factors and inverts that diagonal block, all in
//               shared memory (look-ahead: the next step's diagonal work overlaps the rest of the update);
//               other CTAs: the remaining upper tiles of A(j+1:, j+1:) -= U(j, j+1:)^T U(j, j+1:)
//            --- barrier ---
// then X by doubling over block sizes 64, 128, ...: X12 = -X11 (U12 X22), every tile of a level in parallel.
// A pivot that is not > 0 (or NaN) records kStatusNotSPD with the global column (1-based), LAPACK's info, and every
// CTA leaves at the next barrier.  Every barrier wait is time-limited.
#include <algorithm>
#include <type_traits>

#include "gemm_tile.cuh"
#include "kernels.h"

namespace xtbeig {

namespace {

constexpr int NB = 64;
constexpr int kThreads = kGemmThreads;  // 128: the tile routine's CTA shape

struct PotrfParams {
  double* a;
  int lda;
  double* x;
  int ldx;
  double* t;  // n x n scratch, ld n
  int n;
  unsigned* counter;
  DeviceStatus* st;
  uint64_t limit_ns;
};

constexpr int kLeafLd = NB + 4;  // 4 (mod 16): fragment loads of a half warp hit 16 distinct 8-byte banks
constexpr size_t kLeafElems = (size_t)NB * kLeafLd + NB + 4;  // rows, pivots, row counter and flag
constexpr size_t kSmemBytes = (tile::smem_elems<double>() + kLeafElems) * sizeof(double);
static_assert((size_t)NB * kLeafLd <= tile::smem_elems<double>(), "the panel fits the tile pipeline's region");

// 1 / sqrt(d) for d > 0 without a branch, so that the pivot chain interleaves with the row updates: the hardware's
// approximation y and one third-order step, y (1 + e / 2 + 3 e^2 / 8) with e = 1 - d y^2 (the series of (1 - e)^(-1/2); the
// approximation's error cubed is far below the last bit).  e comes from the exact product d y = p + pl: with p alone its
// rounding was as large as the result's own (0.99 ulp instead of 0.52).  The approximation flushes subnormal arguments,
// so small d are scaled by 2^200 first.
__device__ __forceinline__ double pivot_rsqrt(double d) {
  const bool small = d < 1e-250;
  const double ds = small ? d * 0x1p200 : d;
  double y;
  asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(ds));
  const double p = ds * y, pl = fma(ds, y, -p);
  const double e = fma(-pl, y, fma(-p, y, 1.0));
  const double r = fma(y * e, fma(0.375, e, 0.5), y);
  return small ? r * 0x1p100 : r;
}
// sqrt(d) from r = pivot_rsqrt(d): one Newton step on d r, whose residual is exact except where it would be subnormal.
__device__ __forceinline__ double pivot_sqrt(double d, double r) {
  const double s = d * r;
  return d < 1e-280 ? s : fma(fma(-s, s, d), 0.5 * r, s);
}

// The pivot state of the owner warp, the same in every lane: d = M(k, k), r = 1 / sqrt(d), and the two values the next
// pivot follows from, a = M(k, k+1) and b = M(k+1, k+1): d' = b - (a r)^2 needs no shuffle once r is known.
struct LeafPivot {
  double d, r, a, b;
  double x0, x1;  // the pivot row's entries in this lane's columns
  int bad;        // first pivot of this block that is not > 0
};

// Elimination steps k = 16 b .. 16 b + 15 of the leaf (see leaf_factor_invert) on the 16 rows of one warp: its owner,
// warp b, leaves the final rows in `rows` and counts them in *done, two at a time; the warps below follow.  Both are
// rolled loops of about a hundred instructions: unrolled over the 64 steps the code, run once per leaf, was bound by
// instruction fetch (twice the time).  m holds the sum of the products subtracted so far; the block's own row stays in
// `rows` and joins when it becomes the pivot row, so that an entry is rounded once at the block's magnitude.  With the
// products subtracted from the entry one by one, U^T U was three times as far from S (n = 130: 1.2e-15 against 4.1e-16,
// S(k, k) about 2) and the whole factorization 2 % faster.
// kSecond: column k lies in the lanes' second column.  Q0: first of the 16 steps; ROWS: rows below the pivot that may
// still be unfinished (15 in the first eight steps, 7 in the last eight).
template <bool kSecond, int Q0, int ROWS>
__device__ __forceinline__ void leaf_own_steps(double (&m)[16][2], LeafPivot& v, int blk, double* rows, double* diag,
                                               volatile int* done, int lane) {
  const int l0 = (16 * blk) & 31;
#pragma unroll 1
  for (int q = Q0; q < Q0 + 8; ++q) {
    // The pivot row is m[0]: every update writes its row one place up.
    const int k = 16 * blk + q;
    const bool at = lane == l0 + q;
    const double r = v.r, u1 = v.a * r;
    // The block's own entries of the next row and of the pivot after it (past the last row: unused).
    const int k1 = min(k + 1, NB - 1), k2 = min(k + 2, NB - 1);
    const double n0 = rows[k1 * kLeafLd + lane], n1 = rows[k1 * kLeafLd + lane + 32], nb = rows[k2 * kLeafLd + k2];
    v.bad = (!(v.d > 0.0) && v.bad < 0) ? k : v.bad;
    // U(k, :) right of k, W(k, :) from k to the left.
    const double p0 = (!kSecond && at) ? r : v.x0 * r, p1 = (kSecond && at) ? r : v.x1 * r;
    double* row = rows + k * kLeafLd;
    row[lane] = p0;
    row[lane + 32] = p1;
    if (lane == 0) diag[k] = v.d;
    v.d = fma(-u1, u1, v.b);
    v.r = pivot_rsqrt(v.d);  // beside the row updates
#pragma unroll
    for (int i = 1; i <= ROWS; ++i) {
      // U(k, row k + i); beyond the block: unused
      const double u = i == 1 ? u1 : __shfl_sync(0xffffffffu, kSecond ? p1 : p0, l0 + q + i);
      m[i - 1][0] = fma(-u, p0, (!kSecond && at) ? 0.0 : m[i][0]);  // column k becomes -U(k, row) W(k, k)
      m[i - 1][1] = fma(-u, p1, (kSecond && at) ? 0.0 : m[i][1]);
      if (i == 1) {
        v.x0 = n0 + m[0][0];
        v.x1 = n1 + m[0][1];
      }
      if (i == 3) {
        v.a = __shfl_sync(0xffffffffu, kSecond ? v.x1 : v.x0, l0 + q + 2);
        v.b = nb + __shfl_sync(0xffffffffu, kSecond ? m[1][1] : m[1][0], l0 + q + 2);
      }
    }
    if (q & 1) {
      __syncwarp();
      __threadfence_block();
      if (lane == 0) *done = k + 1;
    }
  }
}

template <bool kSecond>
__device__ __forceinline__ void leaf_own_block(double (&m)[16][2], int blk, double* rows, double* diag,
                                               volatile int* done, int* s_bad, int lane) {
  const int l0 = (16 * blk) & 31;
  const double* row = rows + 16 * blk * kLeafLd;
  LeafPivot v;
  v.x0 = row[lane] + m[0][0];
  v.x1 = row[lane + 32] + m[0][1];
  v.d = __shfl_sync(0xffffffffu, kSecond ? v.x1 : v.x0, l0);
  v.a = __shfl_sync(0xffffffffu, kSecond ? v.x1 : v.x0, l0 + 1);
  v.b = row[16 * blk + 1 + kLeafLd] + __shfl_sync(0xffffffffu, kSecond ? m[1][1] : m[1][0], l0 + 1);
  v.r = pivot_rsqrt(v.d);
  v.bad = -1;
  leaf_own_steps<kSecond, 0, 15>(m, v, blk, rows, diag, done, lane);
  leaf_own_steps<kSecond, 8, 7>(m, v, blk, rows, diag, done, lane);
  if (v.bad >= 0 && lane == 0) atomicMin(s_bad, v.bad);
}

template <bool kSecond>
__device__ __forceinline__ void leaf_follow_steps(double (&m)[16][2], int b, const double* rows, const volatile int* done,
                                                  int warp, int lane, DeviceStatus* st, uint64_t limit_ns, bool& waits) {
#pragma unroll 1
  for (int q = 0; q < 16; ++q) {
    const int k = 16 * b + q;
    if ((q & 1) == 0) {
      // The owner never waits for this warp, so the wait ends.  One that ran out of time has set the status, which the
      // next grid barrier returns on; the rows are then read as they are, without another wait.
      waits = waits && wait_count(done, k + 2, st, limit_ns, k);
      __threadfence_block();
    }
    const bool at = lane == (k & 31);
    const double* row = rows + k * kLeafLd;
    const double p0 = row[lane], p1 = row[lane + 32];
    double u[16];
#pragma unroll
    for (int i = 0; i < 16; i += 2) {
      const double2 t = *reinterpret_cast<const double2*>(row + 16 * warp + i);
      u[i] = t.x;
      u[i + 1] = t.y;
    }
#pragma unroll
    for (int i = 0; i < 16; ++i) {
      m[i][0] = fma(-u[i], p0, (!kSecond && at) ? 0.0 : m[i][0]);
      m[i][1] = fma(-u[i], p1, (kSecond && at) ? 0.0 : m[i][1]);
    }
  }
}

// Factor and invert the nb x nb (nb <= 64) diagonal block at (j0, j0) with the CTA's 128 threads: U in place in a,
// X = U^-1 (upper; x's strict lower part is left as it is) into x.  Returns false (all threads) on a pivot that is
// not > 0, after recording kStatusNotSPD with the global column (1-based).  The frame beyond nb is the identity.
//
// The block is the kernel's critical path, and its chain of 64 pivots is what bounds it.  Factor and inverse come from
// one elimination in registers (warp w holds rows 16 w .. 16 w + 15, lane l columns l and l + 32): with M = [A | I] the
// step of pivot k scales row k by 1 / sqrt(M(k, k)) and subtracts U(k, i) times it from every row i > k.  Left of the
// diagonal the rows then grow W = U^-T, which takes the place of A's lower triangle (at step k column k becomes
// -U(k, i) W(k, k)), so the inverse costs no further step.  The owner warp runs down its 16 rows by shuffles alone,
// leaving each final row in shared memory; the warps below follow it at their own pace (a row counter, no block
// barrier).  One block alone (with its panel update): about 40 k cycles, where panels of 8 columns with block barriers and
// a separate block-wise inverse took 57 k; potrf + inverse n = 130 149 -> 120 us, 619 493 -> 407, 1788 1.42 -> 1.07 ms (of
// which the tiles of the trailing update, gemm_tile, gave a part).
// With a panel (the kp x nb block row U(j0 - kp : j0, j0 : j0 + nb), ld lda), the block's trailing update
// A -= P^T P runs first, by matrix instructions (gsm: the tile pipeline's region, free while the leaf runs, holds P).
__device__ bool leaf_factor_invert(const double* panel, int kp, double* a, int lda, double* x, int ldx, int j0,
                                   int nb, DeviceStatus* st, uint64_t limit_ns, double* smem, double* gsm) {
  double* rows = smem;                      // [64][kLeafLd]
  double* diag = rows + NB * kLeafLd;       // the pivots, then U(k, k)
  int* s_bad = reinterpret_cast<int*>(diag + NB);
  volatile int* done = s_bad + 1;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  __syncthreads();
  // Stage A (rows of the upper triangle) and P, coalesced, every load of a thread in flight at once.
  constexpr int kPer = 32;
  for (int base = 0; base < NB * NB; base += kThreads * kPer) {
    double v[kPer], w[kPer];
#pragma unroll
    for (int t = 0; t < kPer; ++t) {
      const int idx = base + tid + kThreads * t, r = idx % NB, c = idx / NB;
      v[t] = c < nb ? (r <= c ? a[(j0 + r) + (size_t)(j0 + c) * lda] : 0.0) : (r == c ? 1.0 : 0.0);
      w[t] = (panel && r < kp && c < nb) ? panel[r + (size_t)c * lda] : 0.0;
    }
#pragma unroll
    for (int t = 0; t < kPer; ++t) {
      const int idx = base + tid + kThreads * t, r = idx % NB, c = idx / NB;
      rows[r * kLeafLd + c] = v[t];
      if (panel) gsm[r * kLeafLd + c] = w[t];
    }
  }
  if (tid == 0) { *s_bad = NB; *done = 0; }
  __syncthreads();
  if (panel) {
    // A -= P^T P on the upper 8 x 8 tiles with the FP64 matrix instruction: warp w takes tile rows w and 7 - w, nine
    // tiles; lane l holds P(4 kk + l % 4, 8 t + l / 4) of either operand.
    const int kr = lane & 3, cr = lane >> 2;
    double acc[9][2];
#pragma unroll
    for (int t = 0; t < 9; ++t) acc[t][0] = acc[t][1] = 0.0;
    const int rows0 = warp, rows1 = 7 - warp;  // tiles (rows0, rows0 .. 7), then (rows1, rows1 .. 7)
#pragma unroll 4
    for (int kk = 0; kk < NB; kk += 4) {       // rows of P beyond kp are zero
      const double* pk = gsm + (kk + kr) * kLeafLd + cr;
      const double a0 = pk[8 * rows0], a1 = pk[8 * rows1];
#pragma unroll
      for (int t = 0; t < 9; ++t) {
        const bool first = t < 8 - rows0;
        const double bf = pk[8 * (first ? rows0 + t : rows1 + t - (8 - rows0))];
        tile::mma_f64(acc[t], first ? a0 : a1, bf);
      }
    }
#pragma unroll
    for (int t = 0; t < 9; ++t) {
      const bool first = t < 8 - rows0;
      const int r = 8 * (first ? rows0 : rows1) + cr, c = 8 * (first ? rows0 + t : rows1 + t - (8 - rows0)) + 2 * kr;
      double2* dst = reinterpret_cast<double2*>(rows + r * kLeafLd + c);
      double2 v = *dst;
      v.x -= r <= c ? acc[t][0] : 0.0;  // below the diagonal the rows stay zero: W joins them there
      v.y -= r <= c + 1 ? acc[t][1] : 0.0;
      *dst = v;
    }
    __syncthreads();
  }
  double m[16][2];
#pragma unroll
  for (int i = 0; i < 16; ++i) m[i][0] = m[i][1] = 0.0;
  bool waits = true;  // no wait has run out
#pragma unroll 1
  for (int b = 0; b < warp; ++b) {
    if (b < 2) leaf_follow_steps<false>(m, b, rows, done, warp, lane, st, limit_ns, waits);
    else leaf_follow_steps<true>(m, b, rows, done, warp, lane, st, limit_ns, waits);
  }
  if (warp < 2) leaf_own_block<false>(m, warp, rows, diag, done, s_bad, lane);
  else leaf_own_block<true>(m, warp, rows, diag, done, s_bad, lane);
  __syncthreads();
  if (*s_bad < NB) {
    if (tid == 0) set_status(st, kStatusNotSPD, j0 + *s_bad + 1, 0);
    __syncthreads();
    return false;
  }
  if (tid < NB) diag[tid] = pivot_sqrt(diag[tid], rows[tid * kLeafLd + tid]);
  __syncthreads();
#pragma unroll 8
  for (int idx = tid; idx < NB * NB; idx += kThreads) {
    const int r = idx % NB, c = idx / NB;
    if (r <= c && c < nb) {
      a[(j0 + r) + (size_t)(j0 + c) * lda] = r == c ? diag[r] : rows[r * kLeafLd + c];
      x[(j0 + r) + (size_t)(j0 + c) * ldx] = rows[c * kLeafLd + r];  // X(r, c) = W(c, r)
    }
  }
  __syncthreads();
  return true;
}

__device__ __forceinline__ GemmDesc<double> tile_desc(int M, int N, int K, double alpha, const double* A, int lda,
                                                      int transA, const double* B, int ldb, double beta, double* C,
                                                      int ldc, int mode) {
  GemmDesc<double> d{};
  d.A = A; d.B = B; d.C = C;
  d.M = M; d.N = N; d.K = K;
  d.lda = lda; d.ldb = ldb; d.ldc = ldc;
  d.alpha = alpha; d.beta = beta;
  d.transA = transA; d.transB = 0;
  d.mode = mode;
  return d;
}

__global__ void __launch_bounds__(kThreads, 1) potrf_persistent_kernel(PotrfParams p) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  double* gsm = reinterpret_cast<double*>(smem_raw);         // tile pipeline
  double* lsm = gsm + tile::smem_elems<double>();            // leaf block
  const int G = gridDim.x, cta = blockIdx.x, n = p.n;
  const int nt = (n + NB - 1) / NB;
  double* a = p.a;
  double* x = p.x;
  const int lda = p.lda, ldx = p.ldx;
  unsigned epoch = 0;
  if (ld_volatile_i32(&p.st->code) != 0) return;
  auto bsize = [&](int b) { return min(NB, n - b * NB); };

  if (cta == 0) leaf_factor_invert(nullptr, 0, a, lda, x, ldx, 0, bsize(0), p.st, p.limit_ns, lsm, gsm);
  if (!group_barrier(p.counter, (unsigned)G, epoch, p.st, p.limit_ns)) return;
  if (ld_volatile_i32(&p.st->code) != 0) return;

  for (int j = 0; j + 1 < nt; ++j) {
    const int j0 = j * NB, nbj = bsize(j);
    // B: block row U(j, c) = X(j,j)^T A(j, c), in place (each tile reads only its own block of A).
    for (int c = j + 1 + cta; c < nt; c += G) {
      const int c0 = c * NB;
      GemmDesc<double> d = tile_desc(nbj, bsize(c), nbj, 1.0, x + j0 + (size_t)j0 * ldx, ldx, 1,
                                     a + j0 + (size_t)c0 * lda, lda, 0.0, a + j0 + (size_t)c0 * lda, lda, kTriALower);
      tile::gemm_tile<double>(d, 0, 0, gsm);
    }
    // CTA 0's phase C reads only the block-row tile it has just written itself (c = j + 1), so it counts itself in
    // and starts the diagonal block at once; the others wait for every block-row tile.
    if (cta == 0 && G > 1) {
      group_arrive(p.counter, epoch);
    } else if (!group_barrier(p.counter, (unsigned)G, epoch, p.st, p.limit_ns)) {
      return;
    }
    // C: trailing update of the upper tiles (r, c), j < r <= c; CTA 0 takes (j+1, j+1) and then the next diagonal.
    const int m = nt - j - 1;
    if (cta == 0) {
      const int r0 = (j + 1) * NB;
      leaf_factor_invert(a + j0 + (size_t)r0 * lda, nbj, a, lda, x, ldx, r0, bsize(j + 1), p.st, p.limit_ns, lsm, gsm);
    }
    const int ntile = m * (m + 1) / 2 - 1;  // upper tiles of the m x m trailing block, except (j+1, j+1)
    const int workers = G > 1 ? G - 1 : 1;
    const int me = G > 1 ? cta - 1 : 0;
    if (G == 1 || cta > 0) {
      for (int t = me; t < ntile; t += workers) {
        // t -> (rr, cc) over the upper triangle by columns, skipping (0, 0): column cc holds rows 0..cc.
        int q = t + 1, cc = 0;
        while (q > cc) { q -= cc + 1; ++cc; }
        const int rr = q;
        const int r = j + 1 + rr, c = j + 1 + cc;
        const int r0 = r * NB, c0 = c * NB;
        GemmDesc<double> d = tile_desc(bsize(r), bsize(c), nbj, -1.0, a + j0 + (size_t)r0 * lda, lda, 1,
                                       a + j0 + (size_t)c0 * lda, lda, 1.0, a + r0 + (size_t)c0 * lda, lda,
                                       r == c ? kCUpper : 0);
        tile::gemm_tile<double>(d, 0, 0, gsm);
      }
    }
    if (!group_barrier(p.counter, (unsigned)G, epoch, p.st, p.limit_ns)) return;
    if (ld_volatile_i32(&p.st->code) != 0) return;
  }

  // X by doubling over block pairs: T = U12 X22 (scratch t), X12 = -X11 T.
  for (int sz = NB; sz < n; sz *= 2) {
    const int tb = sz / NB;  // blocks per half
    const int pairs = (n + 2 * sz - 1) / (2 * sz);
    // tiles of all pairs: (pair, row block in first half, column block in second half)
    int total = 0;
    for (int pr = 0; pr < pairs; ++pr) {
      const int p0 = pr * 2 * sz, s2 = min(sz, n - p0 - sz);
      if (s2 > 0) total += tb * ((s2 + NB - 1) / NB);
    }
    for (int phase = 0; phase < 2; ++phase) {
      for (int t = cta; t < total; t += G) {
        int rem = t, pr = 0;
        for (;; ++pr) {
          const int p0 = pr * 2 * sz, s2 = min(sz, n - p0 - sz);
          const int cnt = s2 > 0 ? tb * ((s2 + NB - 1) / NB) : 0;
          if (rem < cnt) break;
          rem -= cnt;
        }
        const int p0 = pr * 2 * sz, s2 = min(sz, n - p0 - sz);
        // Long sums first (K grows with the column block in the first product, shrinks with the row block in the
        // second), so that a CTA's second tile is a short one: at n = 1788 the top level's 196 tiles take 148 CTAs 1.3
        // instead of 2 longest tiles' time per product.
        const int ncb = (s2 + NB - 1) / NB;
        const int rb = phase == 0 ? rem % tb : rem / ncb, cb = phase == 0 ? ncb - 1 - rem / tb : rem % ncb;
        const int r0 = p0 + rb * NB, c0 = p0 + sz + cb * NB;
        const int rows = NB, cols = min(NB, p0 + sz + s2 - c0);
        double* tt = p.t + r0 + (size_t)c0 * n;
        if (phase == 0) {
          // T(r0 block, c0 block) = U(r0, p0+sz : p0+sz+s2) X(p0+sz : , c0): K over the second half (X22 upper).
          GemmDesc<double> d = tile_desc(rows, cols, s2, 1.0, a + r0 + (size_t)(p0 + sz) * lda, lda, 0,
                                         x + (p0 + sz) + (size_t)c0 * ldx, ldx, 0.0, tt, n, 0);
          d.mode = 0;
          // X22 is upper triangular: rows of the second half beyond the column block are zero.
          d.K = min(s2, c0 + cols - (p0 + sz));
          tile::gemm_tile<double>(d, 0, 0, gsm);
        } else {
          // X(r0 block, c0 block) = -X(r0, p0 : p0+sz) T(p0 : p0+sz, c0): X11 upper, so K starts at the row block.
          const int k0 = r0 - p0;
          GemmDesc<double> d = tile_desc(rows, cols, sz - k0, -1.0, x + r0 + (size_t)r0 * ldx, ldx, 0,
                                         p.t + r0 + (size_t)c0 * n, n, 0.0, x + r0 + (size_t)c0 * ldx, ldx, 0);
          tile::gemm_tile<double>(d, 0, 0, gsm);
        }
      }
      if (!group_barrier(p.counter, (unsigned)G, epoch, p.st, p.limit_ns)) return;
    }
  }
}

}  // namespace

cudaError_t potrf_inverse_upper(int n, double* a, int lda, double* x, int ldx, double* t, unsigned* counter,
                                int grid, DeviceStatus* st, uint64_t limit_ns, cudaStream_t s) {
  if (n <= 0) return cudaSuccess;
  cudaError_t err = cudaFuncSetAttribute(potrf_persistent_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)kSmemBytes);
  if (err != cudaSuccess) return err;
  if ((err = cudaMemsetAsync(x, 0, sizeof(double) * ((size_t)ldx * (n - 1) + n), s)) != cudaSuccess) return err;
  if ((err = cudaMemsetAsync(counter, 0, 64 * sizeof(unsigned), s)) != cudaSuccess) return err;
  PotrfParams p{a, lda, x, ldx, t, n, counter, st, limit_ns};
  const int nt = (n + NB - 1) / NB;
  // Enough CTAs for the widest phase (the first trailing update), never more than co-resident (one per SM).
  const int G = std::max(1, std::min(grid, std::max(2, nt * (nt - 1) / 2)));
  void* args[] = {(void*)&p};
  err = cudaLaunchCooperativeKernel((void*)potrf_persistent_kernel, dim3(G), dim3(kThreads), args, kSmemBytes, s);
  note_launches();
  return err;
}

}  // namespace xtbeig
