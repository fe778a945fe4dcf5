// Divide and conquer for the symmetric tridiagonal eigenproblem on the device (the contract of LAPACK xstedc with
// COMPZ = 'I', which xtb_dstedc exposes: reference Sources/Diagonalization/Exports.swift:88-115; the reference's own
// merge is Stages/ParallelDivideAndConquer.swift:42-211, a port of LAPACK's dlaed1/2/3).
//
// B200 design.  The recursion is flattened into levels: the tree of tears is fixed by n alone, so every merge of one
// level runs in the same launches (one CTA or warp per merge / root / column).  The subtrees of at most 64 are solved by
// one CTA each in shared memory (dc_subtree_kernel); the levels above them run bottom-up.  Per level:
//   deflate   one CTA per merge: z from the halves' boundary rows, merge-sort of the two ascending eigenvalue lists,
//             small-z deflation (rho |z_i| <= tol) and close-pair deflation by Givens rotation (Dongarra-Sorensen),
//             classification of the surviving columns (upper half only / both / lower half only) so the merge GEMM
//             skips the zero blocks, and the device-side sizes of the two merge GEMMs;
//   rotate    apply the recorded rotations to the eigenvector columns, gather survivors and deflated columns;
//   secular   one warp per root, FP64: lambda_j = dlamda_o + tau with tau relative to the nearer pole (so that
//             dlamda_i - lambda_j is formed without cancellation), iterated with the two-pole rational model of the
//             secular function ("middle way", R.-C. Li 1993) inside a bisection bracket;
//   zhat      one warp per i: Gu and Eisenstat's recomputed z (1995) from the computed roots, which makes the
//             eigenvectors of the rank-one problem numerically orthogonal;
//   vectors   one warp per column: u_j = zhat ./ (dlamda - lambda_j), normalised, rows placed in GEMM order;
//   gemm      two grouped FP64 tensor-core GEMMs per merge (upper rows, lower rows);
//   order     final ascending order of roots and deflated eigenvalues, columns copied into place.
// The tridiagonal is scaled by max(|d|, |e|) first and the eigenvalues scaled back, as xstedc does.  No floating-point
// atomics are used, so results are deterministic.
#include <algorithm>
#include <cstring>
#include <vector>

#include "common.cuh"
#include "kernels.h"

namespace xtbeig {

namespace {

struct MergeDesc {
  int s, n1, n2, pad;
};

struct MergeInfo {
  int K;       // surviving (non-deflated) count
  int c1, c2, c3;
  int nrot;
  int ndefl;
  double rho;
};

struct DcBufs {
  int n;       // total size
  int ld;      // leading dimension of the n x n work matrices (= n)
  double* dd;  // current eigenvalues by position
  double* ee;  // scaled off-diagonal
  double* Qa;  // eigenvectors (input of the level)
  double* Qb;  // eigenvectors (output of the level)
  double* Qc;  // gathered columns: survivors in GEMM order, then deflated
  double* Up;  // rank-one eigenvectors, rows in GEMM order
  double* rtau;  // root j = dlam[rorg[j]] + rtau[j]; dlam_i - lambda_j is formed as (dlam_i - dlam[rorg[j]]) - rtau[j]
  double* sd;  // sorted d (then updated by deflation)
  double* sz;  // sorted z
  double* dlam;  // survivors' poles
  double* zk;    // survivors' z
  double* zh;    // recomputed z
  double* lam;   // roots
  double* dval;  // deflated eigenvalues (position order)
  double* rotc;
  double* rots;
  double* scale;  // [1] max norm of (d, e)
  int* sperm;     // sorted position -> local column
  int* typ;       // column type by sorted position (1: upper only, 2: both, 3: lower only, 4: deflated)
  int* ndl;       // scratch list of non-deflated positions
  int* slotOf;    // survivor index -> GEMM slot
  int* srcCol;    // Qc column -> local source column in Qa
  int* rotI;
  int* rotJ;
  int* rorg;      // root j's origin pole (see rtau)
  int* posMerge;  // global position -> merge index at the current level
  MergeDesc* merges;
  MergeInfo* info;
  GemmDesc<double>* gdesc;  // 2 per merge
  DeviceStatus* st;
};

constexpr double kEps = 1.1102230246251565e-16;
constexpr int kSecularWarps = 4;       // warps per secular root at levels with merges of at least kSecularGroupMin
constexpr int kSecularGroupMin = 512;

// Ordering key: NaN sorts as +inf, so every ranking below is a bijection even on non-finite input (a failed earlier
// stage must never turn into an out-of-range index).
__device__ __forceinline__ double okey(double x) { return x == x ? x : INFINITY; }

// Every level kernel returns at once when an earlier stage (or an earlier kernel of this solve) recorded an error.
#define DC_RETURN_IF_FAILED(B) \
  if (ld_volatile_i32(&(B).st->code) != 0) return;

// ------------------------------------------------------------------------------------------------ set-up kernels

__global__ void dc_scale_kernel(int n, const double* d, const double* e, double* scale) {
  __shared__ double scratch[32];
  double m = 0.0;
  for (int i = threadIdx.x; i < n; i += blockDim.x) m = fmax(m, fabs(d[i]));
  for (int i = threadIdx.x; i < n - 1; i += blockDim.x) m = fmax(m, fabs(e[i]));
  m = block_max(m, scratch);
  if (threadIdx.x == 0) scale[0] = m;
}

// dd = d / scale with every split point torn (LAPACK dlaed0's tear: both neighbours lose |e|), ee = e / scale.
__global__ void dc_init_kernel(int n, const double* d, const double* e, double* dd, double* ee,
                               const double* scale) {
  const double sc = scale[0];
  const double inv = sc > 0.0 ? 1.0 / sc : 1.0;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    double v = d[i] * inv;
    if (i > 0) v -= fabs(e[i - 1] * inv);
    if (i < n - 1) v -= fabs(e[i] * inv);
    dd[i] = v;
    if (i < n - 1) ee[i] = e[i] * inv;
  }
}

// Both ping-pong buffers start as the identity and both eigenvalue buffers as the torn diagonal: a 1 x 1 leaf that no
// merge of the current level covers then reads its initial state from whichever buffer is current.
__global__ void dc_identity_kernel(int n, int ld, double* q, double* qb, const double* dd, double* dnext) {
  size_t total = (size_t)n * n;
  for (size_t idx = (size_t)blockIdx.x * blockDim.x + threadIdx.x; idx < total; idx += (size_t)gridDim.x * blockDim.x) {
    int i = (int)(idx % n), j = (int)(idx / n);
    const double v = (i == j) ? 1.0 : 0.0;
    q[i + (size_t)j * ld] = v;
    qb[i + (size_t)j * ld] = v;
    if (j == 0) dnext[i] = dd[i];
  }
}

// ------------------------------------------------------------------------------------------------ deflate

// Block-wide exclusive scan of four 32-bit counters per thread, two to a word; *total receives the sums.
struct Counts {
  unsigned long long a, b;
};
__device__ Counts block_exscan4(Counts v, Counts* scratch, Counts* total) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  auto warp_scan = [&](Counts x) {
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const unsigned long long ya = __shfl_up_sync(0xffffffffu, x.a, o), yb = __shfl_up_sync(0xffffffffu, x.b, o);
      if (lane >= o) {
        x.a += ya;
        x.b += yb;
      }
    }
    return x;
  };
  const Counts x = warp_scan(v);
  __syncthreads();
  if (lane == 31) scratch[warp] = x;
  __syncthreads();
  const Counts w = warp_scan(lane < nw ? scratch[lane] : Counts{0, 0});
  total->a = __shfl_sync(0xffffffffu, w.a, 31);
  total->b = __shfl_sync(0xffffffffu, w.b, 31);
  const unsigned long long pa = __shfl_sync(0xffffffffu, w.a, max(warp - 1, 0));
  const unsigned long long pb = __shfl_sync(0xffffffffu, w.b, max(warp - 1, 0));
  return Counts{(warp > 0 ? pa : 0) + x.a - v.a, (warp > 0 ? pb : 0) + x.b - v.b};
}

// What bounds it: one CTA's chain of dependent steps (searches, scans, the chain of close pairs), so every array that a
// later step reads again lives in shared memory (kSmem; 32 bytes per position, merges of up to kDeflateSmemMax) and a
// thread owns consecutive positions, which takes one scan for each list however long it is.  With the arrays in global
// memory and five scans per 1024 positions a level took 19 us on average (n = 1788, five levels), now 11.  Larger merges
// keep the arrays in global memory.
constexpr int kDeflateSmemMax = 6400;

template <bool kSmem>
__global__ void __launch_bounds__(1024) dc_deflate_kernel(DcBufs B, int nmerge) {
  extern __shared__ __align__(16) unsigned char deflate_smem[];
  __shared__ double s_red[32];
  __shared__ Counts s_scan[32];
  __shared__ int s_nrot;
  const int mi = blockIdx.x;
  if (mi >= nmerge) return;
  DC_RETURN_IF_FAILED(B)
  const MergeDesc md = B.merges[mi];
  const int s = md.s, n1 = md.n1, n2 = md.n2, n = n1 + n2;
  const size_t ld = B.ld;
  const double beta = B.ee[s + n1 - 1];
  const double rho = 2.0 * fabs(beta);
  const double sgn = beta >= 0.0 ? 1.0 : -1.0;
  const double rs2 = 0.70710678118654752440;
  // Sorted values and z, their columns and types; the values before the sort make room for the lists of candidates.
  double* sd = kSmem ? reinterpret_cast<double*>(deflate_smem) : B.sd + s;
  double* sz = kSmem ? sd + n : B.sz + s;
  const double* dd = kSmem ? sz + n : B.dd + s;
  int* ndl = kSmem ? reinterpret_cast<int*>(sz + n) : B.ndl + s;
  int* clist = kSmem ? ndl + n : B.slotOf + s;  // slotOf's range of this merge is written only further down
  int* sperm = kSmem ? clist + n : B.sperm + s;
  int* typ = kSmem ? sperm + n : B.typ + s;
  const int q = (n + blockDim.x - 1) / blockDim.x;  // positions per thread
  const int p0 = min((int)threadIdx.x * q, n), p1 = min(p0 + q, n);
  Counts tot;

  if (kSmem) {
    // Every entry starts in range: a ranking on non-finite input might leave one unwritten.
    for (int i = threadIdx.x; i < n; i += blockDim.x) {
      sz[n + i] = B.dd[s + i];
      sd[i] = sz[i] = 0.0;
      sperm[i] = typ[i] = 0;
    }
    __syncthreads();
  }
  // z and the merge of the two ascending lists (stable: ties keep the upper half first).
  double dmax = 0.0, zmax = 0.0;
  for (int i = threadIdx.x; i < n; i += blockDim.x) {
    double dv, zv;
    int rank;
    if (i < n1) {
      dv = dd[i];
      zv = B.Qa[(size_t)(s + n1 - 1) + (size_t)(s + i) * ld] * rs2;
      int lo = 0, hi = n2;  // count second-half values < dv
      while (lo < hi) { int m = (lo + hi) >> 1; if (okey(dd[n1 + m]) < okey(dv)) lo = m + 1; else hi = m; }
      rank = i + lo;
    } else {
      const int j = i - n1;
      dv = dd[i];
      zv = sgn * B.Qa[(size_t)(s + n1) + (size_t)(s + i) * ld] * rs2;
      int lo = 0, hi = n1;  // count first-half values <= dv
      while (lo < hi) { int m = (lo + hi) >> 1; if (okey(dd[m]) <= okey(dv)) lo = m + 1; else hi = m; }
      rank = j + lo;
    }
    sd[rank] = dv;
    sz[rank] = zv;
    sperm[rank] = i;
    typ[rank] = i < n1 ? 1 : 3;
    dmax = fmax(dmax, fabs(dv));
    zmax = fmax(zmax, fabs(zv));
  }
  dmax = block_max(dmax, s_red);
  zmax = block_max(zmax, s_red);
  const double tol = 8.0 * kEps * fmax(dmax, zmax);
  __syncthreads();

  // Small-z deflation, then the compacted list of candidates for pair deflation.
  int m = 0;
  {
    unsigned cnt = 0;
    for (int p = p0; p < p1; ++p) {
      if (rho * fabs(sz[p]) > tol) ++cnt;
      else typ[p] = 4;
    }
    int at = (int)block_exscan4(Counts{cnt, 0}, s_scan, &tot).a;
    m = (int)tot.a;
    for (int p = p0; p < p1; ++p)
      if (typ[p] != 4) ndl[at++] = p;
    __syncthreads();
  }
  // The pairs that pass the close-pair test before any rotation, compacted in pair order.
  int nc = 0;
  {
    auto close = [&](int i) {
      const int a = ndl[i], b = ndl[i + 1];
      const double za = sz[a], zb = sz[b];
      const double t = hypot(za, zb);
      const double c = zb / t, sn = -za / t;
      return fabs((sd[b] - sd[a]) * c * sn) <= tol;
    };
    unsigned cnt = 0;
    unsigned long long flags = 0;  // of the first 64 of the thread's pairs; later ones are tested again
    for (int i = p0; i < p1 && i < m - 1; ++i)
      if (close(i)) {
        ++cnt;
        if (i - p0 < 64) flags |= 1ull << (i - p0);
      }
    int at = (int)block_exscan4(Counts{cnt, 0}, s_scan, &tot).a;
    nc = (int)tot.a;
    if (cnt > 0)
      for (int i = p0; i < p1 && i < m - 1; ++i)
        if (i - p0 < 64 ? (flags >> (i - p0)) & 1 : close(i)) clist[at++] = i;
    __syncthreads();
  }

  // Sequential chain of close-pair deflations (rare; the test of pair i uses the survivor of pair i-1).  Thread 0
  // visits only the candidates: from each one not yet examined it tests pairs i, i+1, ... until one does not
  // deflate, which is the order and the set of tests of a scan over every pair.
  if (threadIdx.x == 0) {
    int nrot = 0, next = 0;
    for (int w = 0; w < nc; ++w) {
      int i = clist[w];
      if (i < next) continue;
      for (; i < m - 1; ++i) {
        const int a = ndl[i], b = ndl[i + 1];
        const double za = sz[a], zb = sz[b];
        const double t = hypot(za, zb);
        const double c = zb / t, sn = -za / t;
        const double da = sd[a], db = sd[b];
        if (!(fabs((db - da) * c * sn) <= tol)) break;
        sz[b] = t;
        sz[a] = 0.0;
        sd[a] = da * c * c + db * sn * sn;
        sd[b] = da * sn * sn + db * c * c;
        if (typ[a] != typ[b]) typ[b] = 2;
        typ[a] = 4;
        B.rotI[s + nrot] = sperm[a];
        B.rotJ[s + nrot] = sperm[b];
        B.rotc[s + nrot] = c;
        B.rots[s + nrot] = sn;
        ++nrot;
      }
      next = i + 1;
    }
    s_nrot = nrot;
  }
  __syncthreads();

  // Survivors in position order (their values ascend), their type-grouped GEMM slots, deflated list: one scan of the
  // four types' counts.
  unsigned cnt[4] = {0, 0, 0, 0};
  for (int p = p0; p < p1; ++p) {
    const int ty = min(max(typ[p], 1), 4);
#pragma unroll
    for (int t = 0; t < 4; ++t) cnt[t] += ty == t + 1;
  }
  const Counts mine{cnt[0] | (unsigned long long)cnt[1] << 32, cnt[2] | (unsigned long long)cnt[3] << 32};
  const Counts pre = block_exscan4(mine, s_scan, &tot);
  const int c1 = (int)(unsigned)tot.a, c2 = (int)(tot.a >> 32), c3 = (int)(unsigned)tot.b, nd = (int)(tot.b >> 32);
  const int K = c1 + c2 + c3;
  int at1 = (int)(unsigned)pre.a, at2 = (int)(pre.a >> 32), at3 = (int)(unsigned)pre.b, atd = (int)(pre.b >> 32);
  for (int p = p0; p < p1; ++p) {
    const int ty = min(max(typ[p], 1), 4);
    if (ty == 4) {
      B.dval[s + atd] = sd[p];
      B.srcCol[s + K + atd] = sperm[p];
      ++atd;
      continue;
    }
    const int i = at1 + at2 + at3;
    const int slot = ty == 1 ? at1++ : ty == 2 ? c1 + at2++ : c1 + c2 + at3++;
    B.dlam[s + i] = sd[p];
    B.zk[s + i] = sz[p];
    B.slotOf[s + i] = slot;
    B.srcCol[s + slot] = sperm[p];
  }

  if (threadIdx.x == 0) {
    MergeInfo inf;
    inf.K = K; inf.c1 = c1; inf.c2 = c2; inf.c3 = c3; inf.nrot = s_nrot; inf.ndefl = nd; inf.rho = rho;
    B.info[mi] = inf;
    // Merge GEMMs: Qnew(upper rows) = Qc(upper, slots [0, c1+c2)) Up(slots [0, c1+c2), 0:K);
    //              Qnew(lower rows) = Qc(lower, slots [c1, K))     Up(slots [c1, K), 0:K).   Qnew overwrites Qa.
    GemmDesc<double>& gt = B.gdesc[2 * mi];
    GemmDesc<double>& gb = B.gdesc[2 * mi + 1];
    gt.A = B.Qc + (size_t)s + (size_t)s * ld;
    gt.B = B.Up + (size_t)s + (size_t)s * ld;
    gt.C = B.Qa + (size_t)s + (size_t)s * ld;
    gt.M = n1; gt.N = K; gt.K = c1 + c2;
    gb.A = B.Qc + (size_t)(s + n1) + (size_t)(s + c1) * ld;
    gb.B = B.Up + (size_t)(s + c1) + (size_t)s * ld;
    gb.C = B.Qa + (size_t)(s + n1) + (size_t)s * ld;
    gb.M = n2; gb.N = K; gb.K = c2 + c3;
  }
}

// ------------------------------------------------------------------------------------------------ rotate + gather

// grid (merges, row blocks); one thread per row applies the merge's recorded rotations in order (rows are independent).
__global__ void dc_rotate_kernel(DcBufs B) {
  DC_RETURN_IF_FAILED(B)
  const int mi = blockIdx.x;
  const MergeInfo inf = B.info[mi];
  if (inf.nrot == 0) return;
  const MergeDesc md = B.merges[mi];
  const int s = md.s, n = md.n1 + md.n2;
  const size_t ld = B.ld;
  const int r = blockIdx.y * blockDim.x + threadIdx.x;
  if (r >= n) return;
  double* qrow = B.Qa + (size_t)(s + r) + (size_t)s * ld;  // element (r, c) at qrow[c * ld]
  for (int t = 0; t < inf.nrot; ++t) {
    const int i = B.rotI[s + t], j = B.rotJ[s + t];
    const double c = B.rotc[s + t], sn = B.rots[s + t];
    const double qi = qrow[(size_t)i * ld], qj = qrow[(size_t)j * ld];
    qrow[(size_t)i * ld] = c * qi + sn * qj;
    qrow[(size_t)j * ld] = -sn * qi + c * qj;
  }
}

// grid (merges, row blocks of blockDim.x, column chunks of 32): columns gathered into Qc in GEMM slot order.
__global__ void dc_gather_kernel(DcBufs B) {
  DC_RETURN_IF_FAILED(B)
  const int mi = blockIdx.x;
  const MergeDesc md = B.merges[mi];
  const int s = md.s, n = md.n1 + md.n2;
  const int r = blockIdx.y * blockDim.x + threadIdx.x;
  const int c0 = blockIdx.z * 32;
  if (r >= n || c0 >= n) return;
  const size_t ld = B.ld;
  const double* qrow = B.Qa + (size_t)(s + r) + (size_t)s * ld;
  double* crow = B.Qc + (size_t)(s + r) + (size_t)s * ld;
  const int c1 = min(c0 + 32, n);
  // All 32 loads before the first store: the stores could alias the loads for all the compiler knows, so a plain loop
  // would wait one memory latency per column.
  double v[32];
#pragma unroll
  for (int k = 0; k < 32; ++k) v[k] = c0 + k < c1 ? qrow[(size_t)B.srcCol[s + c0 + k] * ld] : 0.0;
#pragma unroll
  for (int k = 0; k < 32; ++k)
    if (c0 + k < c1) crow[(size_t)(c0 + k) * ld] = v[k];
}

// ------------------------------------------------------------------------------------------------ secular equation

// The divisions below are common.cuh's rcp_normal and div_normal: their divisors, differences of poles and roots, are at
// least about 1e-31 of the scaled spectrum, and bad input gives a NaN, as it would by any division.

// Sums over the poles left of the root (psi <= 0), right of it (phi >= 0) and their derivatives; the sum of the terms'
// absolute values is phi - psi.
struct SecSums {
  double psi, dpsi, phi, dphi;
};

// Threads per root: WPR warps, or eight lanes (WPR 0).
template <int WPR>
constexpr int kRootThreads = WPR == 0 ? 8 : 32 * WPR;

// A root is solved by WPR warps together (one CTA of 32 WPR threads when WPR > 1) or by eight lanes: every sum runs over
// the poles strided by the group's threads, then across its warps in warp order through shared memory (sh: 2 x 5 x WPR
// doubles, alternating by `tog`, so one __syncthreads per sum; every thread receives the same value).  The groups of
// eight of a warp may diverge.
template <int WPR>
__device__ __forceinline__ void group_sums(double* v, int cnt, double* sh, int& tog) {
  if constexpr (WPR == 0) {
    const unsigned mask = 0xffu << (threadIdx.x & 24);
#pragma unroll 5
    for (int j = 0; j < cnt; ++j) {
      v[j] += __shfl_xor_sync(mask, v[j], 4);
      v[j] += __shfl_xor_sync(mask, v[j], 2);
      v[j] += __shfl_xor_sync(mask, v[j], 1);
    }
    return;
  }
#pragma unroll 5
  for (int j = 0; j < cnt; ++j) v[j] = warp_sum(v[j]);
  if constexpr (WPR > 1) {
    double* buf = sh + tog * 5 * WPR;
    tog ^= 1;
    const int w = threadIdx.x >> 5;
    if ((threadIdx.x & 31) == 0)
      for (int j = 0; j < cnt; ++j) buf[j * WPR + w] = v[j];
    __syncthreads();
    for (int j = 0; j < cnt; ++j) {
      double r = 0.0;
#pragma unroll
      for (int q = 0; q < WPR; ++q) r += buf[j * WPR + q];
      v[j] = r;
    }
  }
}

template <int WPR>
__device__ __forceinline__ SecSums sec_eval(const double* dl, const double* z, int K, int o, int a, double tau,
                                            double* sh, int& tog) {
  const int lane = threadIdx.x & (kRootThreads<WPR> - 1);
  SecSums r{0, 0, 0, 0};
  const double dlo = dl[o];
#pragma unroll 4
  for (int i = lane; i < K; i += kRootThreads<WPR>) {
    const double del = (dl[i] - dlo) - tau;
    const double inv = rcp_normal(del);
    const double t = z[i] * z[i] * inv, dt = t * inv;
    const bool left = i <= a;
    r.psi += left ? t : 0.0;
    r.dpsi += left ? dt : 0.0;
    r.phi += left ? 0.0 : t;
    r.dphi += left ? 0.0 : dt;
  }
  double v[4] = {r.psi, r.dpsi, r.phi, r.dphi};
  group_sums<WPR>(v, 4, sh, tog);
  return SecSums{v[0], v[1], v[2], v[3]};
}

// Root j of 1/rho + sum_i z_i^2 / (dl_i - lambda) = 0 (rho > 0, dl ascending): lambda = dl[o] + tau.
// Returns false if it did not converge within the iteration limit (the best iterate is still returned).
template <int WPR>
__device__ bool secular_root(const double* dl, const double* z, int K, double rho, int j, int* o_out,
                             double* tau_out, double* sh) {
  const int lane = threadIdx.x & (kRootThreads<WPR> - 1);
  int tog = 0;
  const double rinv = 1.0 / rho;
  if (K == 1) {
    *o_out = 0;
    *tau_out = rho * z[0] * z[0];
    return true;
  }
  int o, a;
  double lo, hi, tau;
  SecSums S{0, 0, 0, 0};
  // The evaluation at the middle of the interval chooses the origin (the nearer pole) and is the first iterate.
  bool have = false;
  if (j < K - 1) {
    const double gap = dl[j + 1] - dl[j];
    a = j;
    S = sec_eval<WPR>(dl, z, K, j, a, 0.5 * gap, sh, tog);
    have = true;
    if (rinv + S.psi + S.phi >= 0.0) { o = j; lo = 0.0; hi = tau = 0.5 * gap; }
    else { o = j + 1; lo = tau = -0.5 * gap; hi = 0.0; }
  } else {
    double zz = 0.0;
    for (int i = lane; i < K; i += kRootThreads<WPR>) zz += z[i] * z[i];
    group_sums<WPR>(&zz, 1, sh, tog);
    o = K - 1;
    lo = 0.0;
    hi = rho * zz;
    a = K - 2;
    tau = 0.5 * (lo + hi);
  }
  const int b = a + 1;
  const double dlo = dl[o];
  const double pa = dl[a] - dlo, pb = dl[b] - dlo;  // poles relative to the origin
  bool conv = false;
  for (int it = 0; it < 120; ++it) {
    if (!have) S = sec_eval<WPR>(dl, z, K, o, a, tau, sh, tog);
    const double f = rinv + S.psi + S.phi;
    const double errb = 8.0 * kEps * (rinv + (S.phi - S.psi)) + kEps * fabs(tau) * (S.dpsi + S.dphi);
    if (!have && fabs(f) <= errb) { conv = true; break; }
    have = false;
    if (f < 0.0) lo = tau; else hi = tau;
    if (hi - lo <= 2.0 * kEps * fmax(fabs(lo), fabs(hi))) { conv = true; break; }
    // Two-pole rational model c + A/(da - eta) + B/(db - eta) matching psi, psi', phi, phi' at tau.
    const double da = pa - tau, db = pb - tau;
    const double A = S.dpsi * da * da, Bm = S.dphi * db * db;
    const double c = f - S.dpsi * da - S.dphi * db;
    const double bq = c * (da + db) + A + Bm, cq = da * db * f;
    double cand1 = NAN, cand2 = NAN;
    if (c == 0.0) {
      if (bq != 0.0) cand1 = div_normal(cq, bq);
    } else {
      double disc = bq * bq - 4.0 * c * cq;
      if (disc < 0.0) disc = 0.0;
      const double sq = sqrt(disc);
      const double big = (bq >= 0.0) ? (bq + sq) : (bq - sq);
      if (big != 0.0) {
        cand1 = div_normal(big, 2.0 * c);
        cand2 = div_normal(2.0 * cq, big);
      }
    }
    double tn = NAN;
    const double e1 = tau + cand1, e2 = tau + cand2;
    const bool ok1 = (e1 > lo) && (e1 < hi), ok2 = (e2 > lo) && (e2 < hi);
    if (ok1 && !ok2) tn = e1;
    else if (ok2 && !ok1) tn = e2;
    else if (ok1 && ok2) tn = fabs(cand1) < fabs(cand2) ? e1 : e2;
    if (!(tn > lo && tn < hi)) tn = 0.5 * (lo + hi);
    if (tn == tau) { conv = true; break; }
    tau = tn;
  }
  *o_out = o;
  *tau_out = tau;
  return conv;
}

// One warp per global position; position s + j of a merge with j < K solves root j.
__global__ void dc_secular_kernel(DcBufs B) {
  const int gw = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (gw >= B.n) return;
  DC_RETURN_IF_FAILED(B)
  const int mi = B.posMerge[gw];
  if (mi < 0) return;
  const MergeDesc md = B.merges[mi];
  const MergeInfo inf = B.info[mi];
  const int s = md.s, j = gw - s, K = inf.K;
  if (j >= K) return;
  const double* dl = B.dlam + s;
  const double* z = B.zk + s;
  int o;
  double tau;
  const bool ok = secular_root<1>(dl, z, K, inf.rho, j, &o, &tau, nullptr);
  if (!ok && lane == 0) set_status(B.st, kStatusSecularNoConv, s + j + 1, s);
  if (lane == 0) {
    B.rorg[s + j] = o;
    B.rtau[s + j] = tau;
    B.lam[s + j] = dl[o] + tau;
  }
}

// The same with WPR warps per root (one CTA per global position), for levels whose merges are large: each evaluation
// of the secular function then loops over K / (32 WPR) poles per thread instead of K / 32.  The early exits depend
// only on the CTA's position (the status word is read once and shared), so all its threads meet every __syncthreads.
template <int WPR>
__global__ void __launch_bounds__(32 * WPR) dc_secular_group_kernel(DcBufs B) {
  __shared__ double sh[2 * 5 * WPR];
  __shared__ int s_failed;
  const int gw = blockIdx.x;
  if (gw >= B.n) return;
  if (threadIdx.x == 0) s_failed = ld_volatile_i32(&B.st->code);
  __syncthreads();
  if (s_failed != 0) return;
  const int mi = B.posMerge[gw];
  if (mi < 0) return;
  const MergeDesc md = B.merges[mi];
  const MergeInfo inf = B.info[mi];
  const int s = md.s, j = gw - s, K = inf.K;
  if (j >= K) return;
  const double* dl = B.dlam + s;
  const double* z = B.zk + s;
  int o;
  double tau;
  const bool ok = secular_root<WPR>(dl, z, K, inf.rho, j, &o, &tau, sh);
  if (threadIdx.x == 0) {
    if (!ok) set_status(B.st, kStatusSecularNoConv, s + j + 1, s);
    B.rorg[s + j] = o;
    B.rtau[s + j] = tau;
    B.lam[s + j] = dl[o] + tau;
  }
}

// One warp per survivor i: zhat_i^2 = -prod_j (dl_i - lambda_j) / prod_{j != i} (dl_i - dl_j)  (Gu-Eisenstat), with
// dl_i - lambda_j formed from root j's origin pole and offset as (dl_i - dl_o) - tau_j, accurate near the pole.
__global__ void dc_zhat_kernel(DcBufs B) {
  const int gw = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (gw >= B.n) return;
  DC_RETURN_IF_FAILED(B)
  const int mi = B.posMerge[gw];
  if (mi < 0) return;
  const MergeDesc md = B.merges[mi];
  const MergeInfo inf = B.info[mi];
  const int s = md.s, i = gw - s, K = inf.K;
  if (i >= K) return;
  const double* dl = B.dlam + s;
  const double di = dl[i];
  double prod = 1.0;
#pragma unroll 4
  for (int j = lane; j < K; j += 32) {
    const double del = (di - dl[B.rorg[s + j]]) - B.rtau[s + j];
    prod *= (j == i) ? -del : div_normal(del, j == i ? 1.0 : di - dl[j]);
  }
  prod = warp_prod(prod);
  if (lane == 0) {
    const double mag = sqrt(fmax(prod, 0.0));
    B.zh[s + i] = copysign(mag, B.zk[s + i]);
  }
}

// One warp per root j: column j of the rank-one problem's eigenvectors, rows in GEMM slot order.
__global__ void dc_vectors_kernel(DcBufs B) {
  const int gw = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (gw >= B.n) return;
  DC_RETURN_IF_FAILED(B)
  const int mi = B.posMerge[gw];
  if (mi < 0) return;
  const MergeDesc md = B.merges[mi];
  const MergeInfo inf = B.info[mi];
  const int s = md.s, j = gw - s, K = inf.K;
  if (j >= K) return;
  const size_t ld = B.ld;
  double* up = B.Up + (size_t)s + (size_t)(s + j) * ld;
  if (K == 1) {
    if (lane == 0) up[B.slotOf[s]] = 1.0;
    return;
  }
  const double* dl = B.dlam + s;
  const double dlo = dl[B.rorg[s + j]], tau = B.rtau[s + j];
  double ss = 0.0;
#pragma unroll 4
  for (int i = lane; i < K; i += 32) {
    const double u = div_normal(B.zh[s + i], (dl[i] - dlo) - tau);
    ss += u * u;
  }
  ss = warp_sum(ss);
  const double inv = 1.0 / sqrt(ss);
#pragma unroll 4
  for (int i = lane; i < K; i += 32) up[B.slotOf[s + i]] = div_normal(B.zh[s + i], (dl[i] - dlo) - tau) * inv;
}

// ------------------------------------------------------------------------------------------------ small subtrees

constexpr int kSubMax = 64;    // largest subtree solved by one CTA
constexpr int kSubLeaf = 8;    // its leaves, diagonalised by Jacobi, one warp each
constexpr int kSubThreads = 512;  // eight lanes per position
constexpr int kSubLd = kSubMax + 1;

// Depth of the tree of halvings at which the largest block (the larger half, repeatedly) is at most `size`.
__host__ __device__ inline int tree_depth(int n, int size) {
  int d = 0;
  while (n > size) {
    n -= n / 2;
    ++d;
  }
  return d;
}
// Block i at depth `depth` of the tree over [lo, hi): the bits of i choose the halves, most significant first, with the
// split of build_levels.
__host__ __device__ inline void tree_block(int i, int depth, int& lo, int& hi) {
  for (int l = depth - 1; l >= 0; --l) {
    const int mid = lo + (hi - lo) / 2;
    if ((i >> l) & 1) lo = mid;
    else hi = mid;
  }
}

struct SubShared {
  double q[2][kSubMax][kSubLd];  // eigenvectors of the current blocks, and those of the next level
  double u[kSubMax][kSubLd];     // rank-one eigenvectors, row = survivor
  double d[2][kSubMax];          // eigenvalues by position
  double e[kSubMax];             // off-diagonal (scaled)
  double sd[kSubMax], sz[kSubMax];                // sorted d and z of a merge
  double dl[kSubMax], zk[kSubMax], zh[kSubMax];   // survivors' poles, z, recomputed z
  double tau[kSubMax], lam[kSubMax], dv[kSubMax]; // roots, deflated values
  double rc[kSubMax], rs[kSubMax];                // rotations
  int perm[kSubMax], flag[kSubMax], nd[kSubMax], cand[kSubMax];
  int col[kSubMax], dcol[kSubMax], org[kSubMax], out[kSubMax], ri[kSubMax], rj[kSubMax];
  int K[4], nrot[4];
  double rho[4];
};

// Jacobi on the warp's m x m leaf (m <= 8) at local position s: q holds the symmetric block on entry and its
// eigenvectors on exit, d the eigenvalues (ascending).  a: the other q buffer, work space at the same place.
// Round-robin ordering, m / 2 disjoint rotations per round; a rotation's angle from two reciprocal square roots,
// cos 2t = |h| / r, sin 2t = b / r with h = a_qq - a_pp, b = 2 a_pq, r = |(h, b)|, and one Newton step towards
// c^2 + s^2 = 1: without it the half dozen roundings of c and s add up in the vectors, whose orthogonality was 1.6 times as
// far off.
__device__ __forceinline__ void sub_leaf(SubShared& S, double (*q)[kSubLd], double (*a)[kSubLd], double* d, int s, int m) {
  const int lane = threadIdx.x & 31, vr = lane >> 2, vj = lane & 3;  // row vr, columns vj and vj + 4
#pragma unroll
  for (int h = 0; h < 8; h += 4) {
    const int c = vj + h;
    if (vr < m && c < m) {
      a[s + vr][s + c] = q[s + vr][s + c];
      q[s + vr][s + c] = vr == c ? 1.0 : 0.0;
    }
  }
  __syncwarp();
  const int kp = (m + 1) & ~1;
  for (int sweep = 0; sweep < 15 && m > 1; ++sweep) {
    double off = 0.0, dg = 0.0;
#pragma unroll
    for (int h = 0; h < 8; h += 4) {
      const int c = vj + h;
      const double x = (vr < m && c < m) ? a[s + vr][s + c] : 0.0;
      if (vr != c) off = fma(x, x, off);
      else dg = fma(x, x, dg);
    }
    off = warp_sum(off);
    dg = warp_sum(dg);
    // Rotations leave rounding of about eps |a| in each of the m (m - 1) entries, at most some 3e-31 of the diagonal's mass
    // for m = 8; what is dropped here is at most 1e-15 of the leaf's norm.
    if (off <= 1e-30 * dg || off == 0.0) break;
    for (int round = 0; round < kp - 1; ++round) {
      // Lane i < kp / 2 forms rotation i; every lane gets the ones it needs by shuffle.
      auto at = [&](int pos) {
        const int x = round + pos - 1;
        return pos == 0 ? 0 : 1 + (x >= kp - 1 ? x - (kp - 1) : x);
      };
      int p = 0, pq = 0;
      double c = 1.0, sn = 0.0;
      if (lane < kp / 2) {
        p = at(lane);
        pq = at(kp - 1 - lane);
        if (p > pq) { const int x = p; p = pq; pq = x; }
        if (pq < m) {
          const double apq = a[s + p][s + pq];
          const double h = a[s + pq][s + pq] - a[s + p][s + p], b = 2.0 * apq;
          const double r2 = fma(h, h, b * b);
          if (apq != 0.0 && r2 > 1e-290) {
            const double ri = rsqrt(r2);
            const double c2 = fma(0.5 * fabs(h), ri, 0.5);
            const double rc = rsqrt(c2);
            c = c2 * rc;
            sn = copysign(0.5, h) * b * ri * rc;
            const double excess = -0.5 * fma(c, c, fma(sn, sn, -1.0));
            c = fma(excess, c, c);
            sn = fma(excess, sn, sn);
          }
        }
      }
      // Two-sided update by 2 x 2 blocks: lane (i, j) = (lane / 4, lane % 4), pairs i and j, lanes 0 .. 15.
      const int i = (lane >> 2) & 3, j = lane & 3;
      const int pi = __shfl_sync(0xffffffffu, p, i), qi = __shfl_sync(0xffffffffu, pq, i);
      const int pj = __shfl_sync(0xffffffffu, p, j), qj = __shfl_sync(0xffffffffu, pq, j);
      const double ci = __shfl_sync(0xffffffffu, c, i), si = __shfl_sync(0xffffffffu, sn, i);
      const double cj = __shfl_sync(0xffffffffu, c, j), sj = __shfl_sync(0xffffffffu, sn, j);
      const bool on = lane < 16 && i < kp / 2 && j < kp / 2, qi_in = qi < m, qj_in = qj < m;
      double xpp = 0.0, xpq = 0.0, xqp = 0.0, xqq = 0.0;
      if (on) {
        xpp = a[s + pi][s + pj];
        if (qj_in) xpq = a[s + pi][s + qj];
        if (qi_in) xqp = a[s + qi][s + pj];
        if (qi_in && qj_in) xqq = a[s + qi][s + qj];
      }
      // The rotations of the vectors: columns p, q of q, one lane per (row, pair).
      const int vp = __shfl_sync(0xffffffffu, p, vj), vq = __shfl_sync(0xffffffffu, pq, vj);
      const double vc = __shfl_sync(0xffffffffu, c, vj), vs = __shfl_sync(0xffffffffu, sn, vj);
      const bool von = vr < m && vj < kp / 2 && vq < m;
      double vxp = 0.0, vxq = 0.0;
      if (von) {
        vxp = q[s + vr][s + vp];
        vxq = q[s + vr][s + vq];
      }
      __syncwarp();
      if (on) {
        // rows: (p, q) <- (c p - s q, s p + c q), then columns alike
        const double tpp = ci * xpp - si * xqp, tqp = si * xpp + ci * xqp;
        const double tpq = ci * xpq - si * xqq, tqq = si * xpq + ci * xqq;
        a[s + pi][s + pj] = cj * tpp - sj * tpq;
        if (qj_in) a[s + pi][s + qj] = sj * tpp + cj * tpq;
        if (qi_in) a[s + qi][s + pj] = cj * tqp - sj * tqq;
        if (qi_in && qj_in) a[s + qi][s + qj] = sj * tqp + cj * tqq;
      }
      if (von) {
        q[s + vr][s + vp] = vc * vxp - vs * vxq;
        q[s + vr][s + vq] = vs * vxp + vc * vxq;
      }
      __syncwarp();
    }
  }
  // Ascending order (ties by index); the columns of q move through registers.
  double w = 0.0;
  int rank = 0;
  if (lane < m) {
    w = a[s + lane][s + lane];
    for (int t = 0; t < m; ++t) {
      const double o = a[s + t][s + t];
      rank += (okey(o) < okey(w) || (okey(o) == okey(w) && t < lane)) ? 1 : 0;
    }
  }
  double v[2] = {0.0, 0.0};
  int to[2] = {0, 0};
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const int c = vj + 4 * h;
    to[h] = __shfl_sync(0xffffffffu, rank, c);
    if (vr < m && c < m) v[h] = q[s + vr][s + c];
  }
  __syncwarp();
  if (lane < m) d[s + rank] = w;
#pragma unroll
  for (int h = 0; h < 2; ++h)
    if (vr < m && vj + 4 * h < m) q[s + vr][s + to[h]] = v[h];
  // the work block is the next level's output buffer: zero outside what the merges write
#pragma unroll
  for (int h = 0; h < 8; h += 4)
    if (vr < m && vj + h < m) a[s + vr][s + vj + h] = 0.0;
  __syncwarp();
}

// Deflation of one merge (n <= 64) by one warp: the steps of dc_deflate_kernel on two positions per lane.
__device__ __forceinline__ void sub_deflate(SubShared& S, int mi, int s, int n, double dmax) {
  const int lane = threadIdx.x & 31;
  const unsigned full = 0xffffffffu, below = (1u << lane) - 1u;
  double* sd = S.sd + s;
  double* sz = S.sz + s;
  int* flag = S.flag + s;  // 1: deflated
  const double rho = S.rho[mi];
  double zmax = 0.0;
  for (int p = lane; p < n; p += 32) zmax = fmax(zmax, fabs(sz[p]));
  zmax = warp_max(zmax);
  const double tol = 8.0 * kEps * fmax(dmax, zmax);
  // Small-z deflation; the positions kept, in order.
  int mk = 0;
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const int p = lane + 32 * h;
    const bool keep = p < n && rho * fabs(sz[p]) > tol;
    if (p < n) flag[p] = keep ? 0 : 1;
    const unsigned b = __ballot_sync(full, keep);
    if (keep) S.nd[s + mk + __popc(b & below)] = p;
    mk += __popc(b);
  }
  __syncwarp();
  // Pairs that pass the close-pair test before any rotation, then the sequential chain over them.
  int nc = 0;
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const int i = lane + 32 * h;
    bool close = false;
    if (i < mk - 1) {
      const int a = S.nd[s + i], b = S.nd[s + i + 1];
      const double za = sz[a], zb = sz[b], t = hypot(za, zb);
      close = fabs((sd[b] - sd[a]) * (zb / t) * (-za / t)) <= tol;
    }
    const unsigned b = __ballot_sync(full, close);
    if (close) S.cand[s + nc + __popc(b & below)] = i;
    nc += __popc(b);
  }
  __syncwarp();
  int nrot = 0;
  if (lane == 0) {
    int next = 0;
    for (int c = 0; c < nc; ++c) {
      int i = S.cand[s + c];
      if (i < next) continue;
      for (; i < mk - 1; ++i) {
        const int a = S.nd[s + i], b = S.nd[s + i + 1];
        const double za = sz[a], zb = sz[b], t = hypot(za, zb);
        const double cs = zb / t, sn = -za / t, da = sd[a], db = sd[b];
        if (!(fabs((db - da) * cs * sn) <= tol)) break;
        sz[b] = t;
        sz[a] = 0.0;
        sd[a] = da * cs * cs + db * sn * sn;
        sd[b] = da * sn * sn + db * cs * cs;
        flag[a] = 1;
        S.ri[s + nrot] = S.perm[s + a];
        S.rj[s + nrot] = S.perm[s + b];
        S.rc[s + nrot] = cs;
        S.rs[s + nrot] = sn;
        ++nrot;
      }
      next = i + 1;
    }
    S.nrot[mi] = nrot;
  }
  __syncwarp();
  int K = 0, nd = 0;
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const int p = lane + 32 * h;
    const bool in = p < n, gone = in && flag[p] != 0;
    const unsigned bs = __ballot_sync(full, in && !gone), bd = __ballot_sync(full, gone);
    if (in && !gone) {
      const int i = K + __popc(bs & below);
      S.dl[s + i] = sd[p];
      S.zk[s + i] = sz[p];
      S.col[s + i] = S.perm[s + p];
    } else if (gone) {
      const int t = nd + __popc(bd & below);
      S.dv[s + t] = sd[p];
      S.dcol[s + t] = S.perm[s + p];
    }
    K += __popc(bs);
    nd += __popc(bd);
  }
  if (lane == 0) S.K[mi] = K;
}

// New eigenvectors of one merge: columns of roots q(:, col(i)) u(i, j), deflated columns copied.  RT x CT threads, each
// RM x CM outputs (RT RM and CT CM at least the merge's size).
template <int RT, int CT, int RM, int CM>
__device__ __forceinline__ void sub_vectors(const SubShared& S, const double (*q)[kSubLd], double (*t)[kSubLd], int s,
                                            int n, int K, int lt) {
  const int rt = lt / CT, ct = lt % CT;
  double acc[RM][CM];
#pragma unroll
  for (int a = 0; a < RM; ++a)
#pragma unroll
    for (int b = 0; b < CM; ++b) acc[a][b] = 0.0;
  // Rows and columns beyond the merge read in-bounds values (other blocks, zeros) that are not stored.
#pragma unroll 4
  for (int i = 0; i < K; ++i) {
    const int c = s + S.col[s + i];
    double x[RM], y[CM];
#pragma unroll
    for (int a = 0; a < RM; ++a) x[a] = q[min(s + rt + RT * a, kSubMax - 1)][c];
#pragma unroll
    for (int b = 0; b < CM; ++b) y[b] = S.u[s + i][min(s + ct + CT * b, kSubMax - 1)];
#pragma unroll
    for (int a = 0; a < RM; ++a)
#pragma unroll
      for (int b = 0; b < CM; ++b) acc[a][b] = fma(x[a], y[b], acc[a][b]);
  }
#pragma unroll
  for (int b = 0; b < CM; ++b) {
    const int j = ct + CT * b;
    if (j >= n) continue;
    const int c = s + S.out[s + j];
#pragma unroll
    for (int a = 0; a < RM; ++a) {
      const int r = rt + RT * a;
      if (r < n) t[s + r][c] = j < K ? acc[a][b] : q[s + r][s + S.dcol[s + j - K]];
    }
  }
}

// The subtrees at depth `depth` of the tree (at most kSubMax long), one CTA each, from the tridiagonal to their
// eigenvalues and vectors, in shared memory: leaves of at most 8 by Jacobi (one warp each), then up to three levels of
// merges.  At depth l of the subtree the CTA's threads split into 2^l groups of 512 / 2^l, one per merge, with eight
// lanes per position: z and the merged order, deflation (one warp), eight lanes per secular root, recomputed z and vector,
// then the product with the blocks' vectors in register tiles.  The steps and tests are those of the level kernels below.
// What bounds it is latency: a few hundred dependent operations per level, in place of nine launches.  It took the place
// of Jacobi leaves of 16 and the level kernels up to 64: the whole tridiagonal solve 203 -> 59 us at n = 37, 346 -> 193 at
// 130, 548 -> 344 at 412 (with the branch-free divisions; now 59, 177 and 289).  Leaves of 8 because a Jacobi round's
// latency does not depend on the size, and 16 take twice the rounds.
// The subtree's tears are those of its ends and of its leaves' ends.  Results go to dd / dnext and the diagonal block of
// both eigenvector buffers (the entry state of the first level above), or, for the whole matrix (depth 0), straight to
// d_out (unscaled) and z's first m_cols columns.
__global__ void __launch_bounds__(kSubThreads, 1) dc_subtree_kernel(int ntot, int depth, const double* d,
                                                                 const double* e, const double* scale_in,
                                                                 double* dd, double* dnext, double* qa, double* qb, int ld,
                                                                 double* d_out, double* z, int ldz, int m_cols, DeviceStatus* st) {
  extern __shared__ __align__(16) unsigned char sub_smem[];
  SubShared& S = *reinterpret_cast<SubShared*>(sub_smem);
  __shared__ double red[32];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  int lo = 0, hi = ntot;
  tree_block(blockIdx.x, depth, lo, hi);
  const int m = hi - lo;
  if (m <= 0 || m > kSubMax) return;
  const int failed = ld_volatile_i32(&st->code);  // an earlier stage's; another CTA may record one meanwhile
  double sc;
  if (depth == 0) {  // the whole matrix: its scale is found here
    double x = 0.0;
    for (int i = tid; i < ntot; i += kSubThreads) x = fmax(x, fmax(fabs(d[i]), i < ntot - 1 ? fabs(e[i]) : 0.0));
    sc = block_max(x, red);
  } else {
    sc = scale_in[0];
  }
  const double inv = sc > 0.0 ? 1.0 / sc : 1.0;
  for (int t = tid; t < kSubMax * kSubLd; t += kSubThreads) {
    (&S.q[0][0][0])[t] = 0.0;
    (&S.q[1][0][0])[t] = 0.0;
    (&S.u[0][0])[t] = 0.0;
  }
  // Columns start in range: a ranking on non-finite input might leave one unwritten.
  if (tid < kSubMax) S.perm[tid] = S.col[tid] = S.dcol[tid] = S.ri[tid] = S.rj[tid] = S.org[tid] = S.out[tid] = 0;
  if (__syncthreads_or(failed)) return;
  const int L = tree_depth(m, kSubLeaf);
  for (int i = tid; i < m; i += kSubThreads) {
    S.q[0][i][i] = d[lo + i] * inv;
    const double off = lo + i < ntot - 1 ? e[lo + i] * inv : 0.0;
    S.e[i] = off;
    if (i < m - 1) S.q[0][i][i + 1] = S.q[0][i + 1][i] = off;
  }
  __syncthreads();
  {
    int s = 0, t = m;
    tree_block(warp, L, s, t);
    const bool has = warp < (1 << L);
    if (has && lane == 0) {  // tears at both ends (an inner end's neighbour loses the same)
      if (lo + s > 0) S.q[0][s][s] -= fabs(s > 0 ? S.e[s - 1] : e[lo - 1] * inv);
      if (lo + t < ntot) S.q[0][t - 1][t - 1] -= fabs(S.e[t - 1]);
      if (t < m) S.q[0][t - 1][t] = S.q[0][t][t - 1] = 0.0;  // outside every leaf
    }
    __syncthreads();
    if (has) sub_leaf(S, S.q[0], S.q[1], S.d[0], s, t - s);
  }
  __syncthreads();
  int cur = 0;
  for (int lev = L - 1; lev >= 0; --lev) {
    const int tp = kSubThreads >> lev, mi = tid / tp, lt = tid - mi * tp;
    int s = 0, t = m;
    tree_block(mi, lev, s, t);
    const int n = t - s, n1 = n / 2, pos = lt >> 3, g = lt & 7;
    double(*q)[kSubLd] = S.q[cur];
    const double* dc = S.d[cur];
    const double beta = S.e[s + n1 - 1];
    // z and the merged ascending order (ties keep the upper half first).
    if (g == 0 && pos < n) {
      const double rs2 = 0.70710678118654752440;
      const double x = dc[s + pos];
      double zv;
      int b0, b1;
      if (pos < n1) {
        zv = q[s + n1 - 1][s + pos] * rs2;
        b0 = n1; b1 = n;
      } else {
        zv = copysign(1.0, beta) * q[s + n1][s + pos] * rs2;
        b0 = 0; b1 = n1;
      }
      const int base = b0;
      while (b0 < b1) {  // second-half values < x, or first-half values <= x
        const int mid = (b0 + b1) >> 1;
        const double o = okey(dc[s + mid]);
        if (pos < n1 ? o < okey(x) : o <= okey(x)) b0 = mid + 1;
        else b1 = mid;
      }
      const int rank = (pos < n1 ? pos : pos - n1) + b0 - base;
      S.sd[s + rank] = x;
      S.sz[s + rank] = zv;
      S.perm[s + rank] = pos;
    }
    if (lt == 0) S.rho[mi] = 2.0 * fabs(beta);
    __syncthreads();
    if (lt < 32) {
      const double dmax = fmax(fmax(fabs(dc[s]), fabs(dc[s + n1 - 1])), fmax(fabs(dc[s + n1]), fabs(dc[s + n - 1])));
      sub_deflate(S, mi, s, n, dmax);
    }
    __syncthreads();
    const int K = S.K[mi], nrot = S.nrot[mi];
    const double rho = S.rho[mi];
    if (lt < n) {
      double* row = q[s + lt] + s;
      for (int r = 0; r < nrot; ++r) {
        const int i = S.ri[s + r], j = S.rj[s + r];
        const double c = S.rc[s + r], sn = S.rs[s + r], xi = row[i], xj = row[j];
        row[i] = c * xi + sn * xj;
        row[j] = -sn * xi + c * xj;
      }
    }
    const double* dl = S.dl + s;
    if (pos < K) {
      int o;
      double tau;
      const bool ok = secular_root<0>(dl, S.zk + s, K, rho, pos, &o, &tau, nullptr);
      if (g == 0) {
        if (!ok) set_status(st, kStatusSecularNoConv, lo + s + pos + 1, lo + s);
        S.org[s + pos] = o;
        S.tau[s + pos] = tau;
        S.lam[s + pos] = dl[o] + tau;
      }
    }
    __syncthreads();
    const unsigned mask = 0xffu << (tid & 24);
    if (pos < K) {  // recomputed z (Gu-Eisenstat)
      const double di = dl[pos];
      double prod = 1.0;
#pragma unroll 4
      for (int j = g; j < K; j += 8) {
        const double del = (di - dl[S.org[s + j]]) - S.tau[s + j];
        prod *= (j == pos) ? -del : div_normal(del, j == pos ? 1.0 : di - dl[j]);
      }
      prod *= __shfl_xor_sync(mask, prod, 4);
      prod *= __shfl_xor_sync(mask, prod, 2);
      prod *= __shfl_xor_sync(mask, prod, 1);
      if (g == 0) S.zh[s + pos] = copysign(sqrt(fmax(prod, 0.0)), S.zk[s + pos]);
    }
    // Final order: roots, then deflated values.
    if (g == 1 && pos < n) {
      int c;
      double x;
      if (pos < K) {
        x = S.lam[s + pos];
        c = pos;
        for (int r = 0; r < n - K; ++r) c += okey(S.dv[s + r]) < okey(x);
      } else {
        const int w = pos - K;
        x = S.dv[s + w];
        c = 0;
        for (int j = 0; j < K; ++j) c += okey(S.lam[s + j]) <= okey(x);
        for (int r = 0; r < n - K; ++r)
          c += (okey(S.dv[s + r]) < okey(x)) || (okey(S.dv[s + r]) == okey(x) && r < w);
      }
      S.out[s + pos] = c;
      S.d[cur ^ 1][s + c] = x;
    }
    __syncthreads();
    if (pos < K) {  // column pos of the rank-one eigenvectors
      if (K == 1) {
        if (g == 0) S.u[s][s] = 1.0;
      } else {
        const double dlo = dl[S.org[s + pos]], tau = S.tau[s + pos];
        double ss = 0.0;
#pragma unroll 4
        for (int i = g; i < K; i += 8) {
          const double x = div_normal(S.zh[s + i], (dl[i] - dlo) - tau);
          S.u[s + i][s + pos] = x;
          ss = fma(x, x, ss);
        }
        ss += __shfl_xor_sync(mask, ss, 4);
        ss += __shfl_xor_sync(mask, ss, 2);
        ss += __shfl_xor_sync(mask, ss, 1);
        const double norm = 1.0 / sqrt(ss);
        for (int i = g; i < K; i += 8) S.u[s + i][s + pos] *= norm;
      }
    }
    __syncthreads();
    double(*out)[kSubLd] = S.q[cur ^ 1];
    if (lev == 0) sub_vectors<16, 32, 4, 2>(S, q, out, s, n, K, lt);
    else if (lev == 1) sub_vectors<16, 16, 2, 2>(S, q, out, s, n, K, lt);
    else sub_vectors<8, 16, 2, 1>(S, q, out, s, n, K, lt);
    cur ^= 1;
    __syncthreads();
  }
  const double(*q)[kSubLd] = S.q[cur];
  if (depth == 0) {
    const double up = sc > 0.0 ? sc : 1.0;
    for (int i = tid; i < m; i += kSubThreads) d_out[i] = S.d[cur][i] * up;
    for (int t = tid; t < m * m_cols; t += kSubThreads) {
      const int c = t / m, r = t - c * m;
      z[(size_t)r + (size_t)c * ldz] = q[r][c];
    }
    return;
  }
  for (int i = tid; i < m; i += kSubThreads) dd[lo + i] = dnext[lo + i] = S.d[cur][i];
  for (int t = tid; t < m * m; t += kSubThreads) {
    const int c = t / m, r = t - c * m;
    const size_t at = (size_t)(lo + r) + (size_t)(lo + c) * ld;
    qa[at] = qb[at] = q[r][c];
  }
}

// ------------------------------------------------------------------------------------------------ partial top merge

// The top merge when only the eigenvectors of the m_cols smallest eigenvalues are wanted: root j lands at output
// position j + #(deflated values below it), so the roots that land below m_cols are a prefix 0 .. Km-1 of the
// ascending roots.  The merge GEMMs' N (root columns) is cut to Km before they run; every eigenvalue is still formed.
// One CTA; the top level has one merge.
__global__ void __launch_bounds__(1024) dc_partial_kernel(DcBufs B, int m_cols) {
  DC_RETURN_IF_FAILED(B)
  __shared__ int red[32];
  const MergeDesc md = B.merges[0];
  const MergeInfo inf = B.info[0];
  const int s = md.s, n = md.n1 + md.n2, K = inf.K, nd = n - K;
  const double* lam = B.lam + s;
  const double* dv = B.dval + s;
  int below = 0;
  for (int j = threadIdx.x; j < K; j += blockDim.x) {
    const double x = lam[j];
    int c = 0;
    for (int t = 0; t < nd; ++t) c += okey(dv[t]) < okey(x);
    below += (j + c < m_cols) ? 1 : 0;
  }
  below = block_sum(below, red);
  if (threadIdx.x == 0) {
    B.gdesc[0].N = below;
    B.gdesc[1].N = below;
  }
}

// ------------------------------------------------------------------------------------------------ final order

// grid (merges, columns): a CTA takes a column of the merge (root or deflated value), counts how many values lie before it
// in the merged ascending order, and copies the column to that place of the next level's eigenvectors; columns placed from
// col_limit on are not wanted (partial top merge).  The column is loaded while the count runs.  Bound by the copy's
// latency; with the ranks in a kernel of their own the two took 18 us a level on average at n = 1788 (9 at n = 412), now
// 10 (5).
__global__ void __launch_bounds__(256) dc_place_kernel(DcBufs B, double* dnext, int col_limit) {
  DC_RETURN_IF_FAILED(B)
  __shared__ int s_cnt[8];
  constexpr int U = 8;
  const int mi = blockIdx.x;
  const MergeDesc md = B.merges[mi];
  const MergeInfo inf = B.info[mi];
  const int s = md.s, n = md.n1 + md.n2, K = inf.K, nd = n - K;
  const double* lam = B.lam + s;
  const double* dv = B.dval + s;
  const size_t ld = B.ld;
  for (int c = blockIdx.y; c < n; c += gridDim.y) {
    const bool root = c < K;
    const double* __restrict__ from = (root ? B.Qa : B.Qc) + (size_t)s + (size_t)(s + c) * ld;
    double v[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int r = threadIdx.x + 256 * u;
      v[u] = r < n ? from[r] : 0.0;
    }
    const double x = root ? lam[c] : dv[c - K];
    const auto kx = okey(x);
    int cnt = 0;
    if (root) {  // its index among the ascending roots, and the deflated values below it
      for (int t = threadIdx.x; t < nd; t += 256) cnt += okey(dv[t]) < kx;
    } else {     // roots up to it, deflated values below it (ties in index order)
      for (int j = threadIdx.x; j < K; j += 256) cnt += okey(lam[j]) <= kx;
      for (int t = threadIdx.x; t < nd; t += 256) {
        const auto kt = okey(dv[t]);
        cnt += kt < kx || (kt == kx && t < c - K);
      }
    }
    const int rank = (root ? c : 0) + block_sum(cnt, s_cnt);
    if (threadIdx.x == 0) dnext[s + rank] = x;
    if (rank >= col_limit) continue;
    double* __restrict__ to = B.Qb + (size_t)s + (size_t)(s + rank) * ld;
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int r = threadIdx.x + 256 * u;
      if (r < n) to[r] = v[u];
    }
    for (int r = threadIdx.x + 256 * U; r < n; r += 256) to[r] = from[r];
  }
}

__global__ void dc_finish_kernel(int n, int m_cols, const double* dd, const double* scale, double* d_out,
                                 const double* q, int ldq, double* z, int ldz) {
  const double sc = scale[0] > 0.0 ? scale[0] : 1.0;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) d_out[i] = dd[i] * sc;
  const size_t total = (size_t)n * m_cols;
  for (size_t idx = (size_t)blockIdx.x * blockDim.x + threadIdx.x; idx < total; idx += (size_t)gridDim.x * blockDim.x) {
    const int i = (int)(idx % n), j = (int)(idx / n);
    z[i + (size_t)j * ldz] = q[i + (size_t)j * ldq];
  }
}

// ------------------------------------------------------------------------------------------------ host plan

struct Level {
  std::vector<MergeDesc> merges;
};

void build_levels(int s, int n, int depth, std::vector<Level>& levels) {
  if (n <= 1) return;
  const int n1 = n / 2, n2 = n - n1;
  build_levels(s, n1, depth + 1, levels);
  build_levels(s + n1, n2, depth + 1, levels);
  if ((int)levels.size() <= depth) levels.resize(depth + 1);
  levels[depth].merges.push_back(MergeDesc{s, n1, n2, 0});
}

template <typename T>
T* carve(char*& p, size_t count) {
  T* r = reinterpret_cast<T*>(p);
  p += ((count * sizeof(T) + 255) / 256) * 256;
  return r;
}

}  // namespace

size_t stedc_work_bytes(int n) {
  const size_t nn = (size_t)n * n;
  size_t b = 0;
  auto add = [&](size_t bytes) { b += ((bytes + 255) / 256) * 256; };
  add(n * sizeof(double) * 2);         // dd, ee
  for (int i = 0; i < 4; ++i) add(nn * sizeof(double));  // Qa Qb Qc Up
  for (int i = 0; i < 11; ++i) add(n * sizeof(double));  // rtau sd sz dlam zk zh lam dval rotc rots dnext
  add(sizeof(double) * 4);             // scale
  for (int i = 0; i < 8; ++i) add(n * sizeof(int));     // sperm typ ndl slotOf srcCol rotI rotJ rorg
  // per level: posMerge, merges, info, gemm descriptors (levels <= 32)
  add((size_t)32 * n * sizeof(int));
  add((size_t)32 * (n / 2 + 2) * sizeof(MergeDesc));
  add((size_t)(n / 2 + 2) * sizeof(MergeInfo));
  add((size_t)32 * (n + 4) * sizeof(GemmDesc<double>));
  return b;
}

size_t stedc_plan_bytes(int n) {
  size_t b = 0;
  auto add = [&](size_t bytes) { b += ((bytes + 255) / 256) * 256; };
  add((size_t)32 * n * sizeof(int));
  add((size_t)32 * (n / 2 + 2) * sizeof(MergeDesc));
  add((size_t)32 * (n + 4) * sizeof(GemmDesc<double>));
  return b;
}

cudaError_t stedc_device(int n, double* d, double* e, double* z, int ldz, void* work, size_t work_bytes, void* plan,
                         bool upload_plan, void* hstage, size_t hstage_bytes, DeviceStatus* st, cudaStream_t s,
                         int m_cols, int leaf) {
  if (n <= 0) return cudaSuccess;
  if (m_cols <= 0 || m_cols > n) m_cols = n;
  if (work_bytes < stedc_work_bytes(n)) return cudaErrorInvalidValue;
  char* p = reinterpret_cast<char*>(work);
  char* pp = reinterpret_cast<char*>(plan);
  DcBufs B{};
  B.n = n;
  B.ld = n;
  const size_t nn = (size_t)n * n;
  B.dd = carve<double>(p, n);
  B.ee = carve<double>(p, n);
  B.Qa = carve<double>(p, nn);
  B.Qb = carve<double>(p, nn);
  B.Qc = carve<double>(p, nn);
  B.Up = carve<double>(p, nn);
  B.rtau = carve<double>(p, n);
  B.sd = carve<double>(p, n);
  B.sz = carve<double>(p, n);
  B.dlam = carve<double>(p, n);
  B.zk = carve<double>(p, n);
  B.zh = carve<double>(p, n);
  B.lam = carve<double>(p, n);
  B.dval = carve<double>(p, n);
  B.rotc = carve<double>(p, n);
  B.rots = carve<double>(p, n);
  double* dnext = carve<double>(p, n);
  B.scale = carve<double>(p, 4);
  B.sperm = carve<int>(p, n);
  B.typ = carve<int>(p, n);
  B.ndl = carve<int>(p, n);
  B.slotOf = carve<int>(p, n);
  B.srcCol = carve<int>(p, n);
  B.rotI = carve<int>(p, n);
  B.rotJ = carve<int>(p, n);
  B.rorg = carve<int>(p, n);
  B.info = carve<MergeInfo>(p, (size_t)(n / 2 + 2));
  // The plan (per-level position map, merges, merge-GEMM descriptor skeletons) depends on n only and lives in its
  // own buffer, uploaded once per n: a captured graph never reads host staging that a later call rewrites.
  int* posAll = carve<int>(pp, (size_t)32 * n);
  MergeDesc* mergesAll = carve<MergeDesc>(pp, (size_t)32 * (n / 2 + 2));
  GemmDesc<double>* gAll = carve<GemmDesc<double>>(pp, (size_t)32 * (n + 4));
  B.st = st;

  // Host plan: levels bottom-up (deepest first).
  std::vector<Level> levels;
  build_levels(0, n, 0, levels);
  std::reverse(levels.begin(), levels.end());
  const int L = (int)levels.size();
  if (L > 32) return cudaErrorInvalidValue;

  // Stage all static per-level data in one pinned buffer, one upload.
  size_t need = 0;
  std::vector<size_t> offPos(L), offMer(L), offG(L);
  std::vector<int> tiles(L), edges(L);
  for (int l = 0; l < L; ++l) {
    offPos[l] = need; need += (size_t)n * sizeof(int);
    offMer[l] = need; need += levels[l].merges.size() * sizeof(MergeDesc);
    need = (need + 15) & ~size_t(15);
    offG[l] = need; need += 2 * levels[l].merges.size() * sizeof(GemmDesc<double>);
  }
  if (upload_plan && need > hstage_bytes) return cudaErrorInvalidValue;
  char* h = reinterpret_cast<char*>(hstage);
  for (int l = 0; l < L; ++l) {
    const auto& ms = levels[l].merges;
    int* pos = upload_plan ? reinterpret_cast<int*>(h + offPos[l]) : nullptr;
    if (pos) {
      for (int i = 0; i < n; ++i) pos[i] = -1;  // -1: an unmerged leaf at this level
      std::memcpy(h + offMer[l], ms.data(), ms.size() * sizeof(MergeDesc));
    }
    GemmDesc<double>* g = upload_plan ? reinterpret_cast<GemmDesc<double>*>(h + offG[l]) : nullptr;
    long tiles64 = 0, tiles32 = 0;
    for (const auto& m : ms) {
      tiles64 += gemm_tiles(m.n1, m.n1 + m.n2, 64) + gemm_tiles(m.n2, m.n1 + m.n2, 64);
      tiles32 += gemm_tiles(m.n1, m.n1 + m.n2, 32) + gemm_tiles(m.n2, m.n1 + m.n2, 32);
    }
    const int edge = edges[l] = gemm_tile_edge<double>(tiles64, tiles32);
    int tb = 0;
    for (size_t mi = 0; mi < ms.size(); ++mi) {
      if (pos)
        for (int i = 0; i < ms[mi].n1 + ms[mi].n2; ++i) pos[ms[mi].s + i] = (int)mi;
      const int nmax = ms[mi].n1 + ms[mi].n2;
      for (int half = 0; half < 2; ++half) {
        const int mrows = half == 0 ? ms[mi].n1 : ms[mi].n2;
        const int tm = (mrows + edge - 1) / edge, tn = (nmax + edge - 1) / edge;
        if (g) {
          GemmDesc<double>& gd = g[2 * mi + half];
          std::memset(&gd, 0, sizeof(gd));
          gd.lda = n; gd.ldb = n; gd.ldc = n;
          gd.alpha = 1.0; gd.beta = 0.0;
          gd.transA = 0; gd.transB = 0; gd.mode = 0;
          gd.tiles_m = tm;
          gd.tiles_n = tn;
          gd.tile_begin = tb;
        }
        tb += tm * tn;
      }
    }
    tiles[l] = tb;
  }
  // Device copies of the plan: posMerge / merges / gemm descriptor skeletons per level, once per n.
  cudaError_t err;
  for (int l = 0; upload_plan && l < L; ++l) {
    const auto& ms = levels[l].merges;
    err = cudaMemcpyAsync(posAll + (size_t)l * n, h + offPos[l], (size_t)n * sizeof(int), cudaMemcpyHostToDevice, s);
    if (err != cudaSuccess) return err;
    err = cudaMemcpyAsync(mergesAll + (size_t)l * (n / 2 + 2), h + offMer[l], ms.size() * sizeof(MergeDesc),
                          cudaMemcpyHostToDevice, s);
    if (err != cudaSuccess) return err;
    err = cudaMemcpyAsync(gAll + (size_t)l * (n + 4), h + offG[l], 2 * ms.size() * sizeof(GemmDesc<double>),
                          cudaMemcpyHostToDevice, s);
    if (err != cudaSuccess) return err;
  }

  err = allow_max_dynamic_smem(dc_deflate_kernel<true>);
  if (err != cudaSuccess) return err;
  // With leaves, the levels at the subtree depth and below are one launch (for n <= kSubMax the whole solve is).
  const int D = leaf > 1 ? tree_depth(n, kSubMax) : -1;
  int l_first = 0;
  if (D >= 0) {
    err = allow_max_dynamic_smem(dc_subtree_kernel);
    if (err != cudaSuccess) return err;
  }
  if (D == 0) {
    dc_subtree_kernel<<<1, kSubThreads, sizeof(SubShared), s>>>(n, 0, d, e, nullptr, nullptr, nullptr, nullptr, nullptr, 0, d,
                                                                z, ldz, m_cols, st);
    note_launches();
    return cudaGetLastError();
  }
  // Index arrays start at 0: an entry that a ranking on non-finite input might leave unwritten stays in range.
  err = cudaMemsetAsync(B.sperm, 0, (size_t)((char*)(B.rorg + n) - (char*)B.sperm), s);
  if (err != cudaSuccess) return err;
  dc_scale_kernel<<<1, 1024, 0, s>>>(n, d, e, B.scale); note_launches();
  dc_init_kernel<<<(n + 255) / 256, 256, 0, s>>>(n, d, e, B.dd, B.ee, B.scale); note_launches();
  {
    const int blocks = (int)std::min<size_t>((nn + 255) / 256, 4096);
    dc_identity_kernel<<<blocks, 256, 0, s>>>(n, n, B.Qa, B.Qb, B.dd, dnext); note_launches();
  }
  if (D > 0) {
    dc_subtree_kernel<<<1 << D, kSubThreads, sizeof(SubShared), s>>>(n, D, d, e, B.scale, B.dd, dnext, B.Qa, B.Qb, n, nullptr,
                                                                     nullptr, 0, 0, st);
    note_launches();
    l_first = std::max(0, L - D);  // levels[l] holds the merges at depth L - 1 - l
  }
  for (int l = l_first; l < L; ++l) {
    const int nm = (int)levels[l].merges.size();
    int maxn = 0;
    for (const auto& m : levels[l].merges) maxn = std::max(maxn, m.n1 + m.n2);
    B.posMerge = posAll + (size_t)l * n;
    B.merges = mergesAll + (size_t)l * (n / 2 + 2);
    B.gdesc = gAll + (size_t)l * (n + 4);
    const int dthreads = maxn > 512 ? 1024 : (maxn > 128 ? 512 : 128);
    if (maxn <= kDeflateSmemMax) {
      dc_deflate_kernel<true><<<nm, dthreads, (size_t)32 * maxn, s>>>(B, nm);
    } else {
      dc_deflate_kernel<false><<<nm, dthreads, 0, s>>>(B, nm);
    }
    note_launches();
    dc_rotate_kernel<<<dim3(nm, (maxn + 127) / 128), 128, 0, s>>>(B); note_launches();
    dc_gather_kernel<<<dim3(nm, (maxn + 127) / 128, (maxn + 31) / 32), 128, 0, s>>>(B); note_launches();
    const int warps_per_block = 8;
    const int nblk = (n + warps_per_block - 1) / warps_per_block;
    if (maxn >= kSecularGroupMin) {
      dc_secular_group_kernel<kSecularWarps><<<n, 32 * kSecularWarps, 0, s>>>(B); note_launches();
    } else {
      dc_secular_kernel<<<nblk, 32 * warps_per_block, 0, s>>>(B); note_launches();
    }
    dc_zhat_kernel<<<nblk, 32 * warps_per_block, 0, s>>>(B); note_launches();
    dc_vectors_kernel<<<nblk, 32 * warps_per_block, 0, s>>>(B); note_launches();
    const bool partial = l == L - 1 && m_cols < n;  // the top merge forms only the wanted columns
    if (partial) {
      dc_partial_kernel<<<1, 1024, 0, s>>>(B, m_cols); note_launches();
    }
    err = gemm_grouped_launch<double>(B.gdesc, 2 * nm, tiles[l], edges[l], s);
    if (err != cudaSuccess) return err;
    dc_place_kernel<<<dim3(nm, std::min(maxn, 65535)), 256, 0, s>>>(B, dnext, partial ? m_cols : n);
    note_launches();
    err = cudaGetLastError();
    if (err != cudaSuccess) return err;
    // Next level reads (dd, Qa) = (dnext, Qb); the old Qa becomes the next output buffer.
    std::swap(B.Qa, B.Qb);
    std::swap(B.dd, dnext);
  }
  dc_finish_kernel<<<1024, 256, 0, s>>>(n, m_cols, B.dd, B.scale, d, B.Qa, n, z, ldz); note_launches();
  return cudaGetLastError();
}

}  // namespace xtbeig
