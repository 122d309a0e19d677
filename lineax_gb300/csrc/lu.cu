// LU factorisation with partial pivoting (getrf) and the matching solve
// (getrs), FP64, row-major.
//
// Two factor paths share one arithmetic definition, the unblocked
// right-looking recurrence of LAPACK getf2:
//   p      = first row of max |a(i,k)|, i >= k            (idamax)
//   swap rows k and p (whole row)
//   a(i,k) = a(i,k) * (1/a(k,k))   (a(i,k) / a(k,k) when |a(k,k)| < DBL_MIN)
//   a(i,j) = fma(-a(i,k), a(k,j), a(i,j))   for i > k, j > k, k ascending
//
//  * n <= kSmallMax: one CTA per matrix, the matrix resident in shared memory.
//  * larger n: right-looking blocked LU with a panel of kNB columns (panel
//    getf2 on a thread-block cluster, then the row interchanges of the other
//    columns with the TRSM of the block row, and a GEMM for the trailing
//    matrix).  The TRSM and the GEMM apply
//    their updates to each element as an FMA chain over k in ascending order
//    starting from the stored value, which is exactly the operation sequence
//    getf2 applies to that element, so both paths give bit-identical factors
//    and pivots for the same input.
#include <cooperative_groups.h>
#include <float.h>
#include <limits.h>

#include "common.cuh"
#include "swaps.cuh"
#include "trisolve.cuh"

namespace lxgb {

constexpr int kSmallMax = 168;   // 168*169*8 B = 227 KB of shared memory
constexpr int kSmallThreads = 256;
constexpr int kSmallMaxThreads = 512;
constexpr size_t kSmSharedBytes = 228 * 1024;   // of an SM, with 1 KB and the static part per CTA
constexpr int kSmallBlocks = (kSmallMax + 31) / 32;
constexpr int kNB = 32;          // panel width of the blocked path
constexpr int kPanelThreads = 1024;

__device__ __forceinline__ double scale_pivot(double v, double akk, double r, bool use_recip) {
  return use_recip ? v * r : v / akk;
}

// ---------------------------------------------------------------------------
// n <= kSmallMax: one CTA per matrix, matrix in shared memory (row stride ld,
// odd so that column walks hit distinct banks).
//
// Warp 0 carries the chain of pivots with the current column in its registers
// (row 32 m + lane in register m): while the other warps apply step k to columns
// >= k + 2 it applies it to column k + 1, finds that column's first maximum by
// integer reductions, forms the reciprocal and writes the multipliers.  The
// others exchange rows k and p as they go: they read u from row p and leave row
// k's update there.  One barrier per column for the CTA, one among the others.
// Bound by the chain up to n of about 64 — an FMA, the reductions, a division, a
// product and a barrier per column, its FP64 instructions in turn with those of
// the update — and by the FP64 pipe of one SM above (n = 128: 217 us of FMAs).
// Measured (one matrix): 47 us at n = 48, 289 at 128, 566 at 168, against 64, 328
// and 660 with the exchange and the scaling between two barriers.
// ---------------------------------------------------------------------------
// Step k on columns k + 2 .. n - 1, exactly NC chunks of 16, a half warp per row:
// rows i0, i0 + 1, i0 + step, ... > k.  Row p (the pivot, still in its place; p = k
// without an interchange) gives u; where i = p the old row k takes the step and
// goes there, and u goes to row k.  The number of chunks is a template argument
// because a chunk that is only predicated off still costs its FP64 instruction.
// `threads`: those that run this.
template <int NC>
__device__ __forceinline__ void small_update(double* A, int ld, int n, int k, int p, int i0,
                                             int step, int lane, int threads) {
  const int j = k + 2 + (lane & 15);
  const bool last = j + 16 * (NC - 1) < n;   // the other chunks are full
  double u[NC];
#pragma unroll
  for (int c = 0; c < NC; ++c) u[c] = (c + 1 < NC || last) ? A[p * ld + j + 16 * c] : 0.0;
  // every u is read before row p is written
  asm volatile("bar.sync 1, %0;" ::"r"(threads) : "memory");
  for (int ib = i0; ib < n; ib += step) {
    const int i = ib + (lane >> 4);
    const bool in = i < n;
    double* y = A + (in ? i : k) * ld;
    const double* src = (i == p) ? A + k * ld : y;
    const double l = y[k];
    double v[NC];
#pragma unroll
    for (int c = 0; c < NC; ++c) v[c] = (c + 1 < NC || last) ? src[j + 16 * c] : 0.0;
#pragma unroll
    for (int c = 0; c < NC; ++c) v[c] = fma(-l, u[c], v[c]);
#pragma unroll
    for (int c = 0; c < NC; ++c)
      if (in && (c + 1 < NC || last)) y[j + 16 * c] = v[c];
    if (i == p) {
#pragma unroll
      for (int c = 0; c < NC; ++c)
        if (c + 1 < NC || last) A[k * ld + j + 16 * c] = u[c];
    }
  }
}

template <int MAX>
__device__ __forceinline__ void small_update_n(int nc, double* A, int ld, int n, int k, int p,
                                               int i0, int step, int lane, int threads) {
  if constexpr (MAX > 0) {
    if (nc == MAX) small_update<MAX>(A, ld, n, k, p, i0, step, lane, threads);
    else small_update_n<MAX - 1>(nc, A, ld, n, k, p, i0, step, lane, threads);
  }
}

template <int MB>
__global__ void __launch_bounds__(kSmallMaxThreads)
getrf_small_kernel(int n, double* __restrict__ a, int64_t stride_a, int32_t* __restrict__ piv,
                   int64_t stride_piv, int32_t* __restrict__ info) {
  extern __shared__ double smem_lu[];
  __shared__ int s_p[2];               // pivot row of the step (k: no interchange), by parity
  const int ld = n | 1;
  double* A = smem_lu;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int nwarps = blockDim.x >> 5;
  const int b = blockIdx.x;
  double* g = a + (int64_t)b * stride_a;
  int32_t* gp = piv + (int64_t)b * stride_piv;
  constexpr int kLoads = 8;
  for (int e0 = tid; e0 < n * n; e0 += kLoads * (int)blockDim.x) {
    double v[kLoads];
#pragma unroll
    for (int q = 0; q < kLoads; ++q) {
      const int e = e0 + q * (int)blockDim.x;
      v[q] = e < n * n ? g[e] : 0.0;
    }
#pragma unroll
    for (int q = 0; q < kLoads; ++q) {
      const int e = e0 + q * (int)blockDim.x;
      if (e < n * n) A[(e / n) * ld + e % n] = v[q];
    }
  }
  __syncthreads();
  int my_info = 0;
  double x[MB];                        // warp 0: the multipliers of column k
  // Warp 0: x holds column k, rows > k - 1 after step k - 1.  Finds its pivot,
  // exchanges rows k and p, scales, and writes the column.
  auto pivot = [&](int k) {
    unsigned long long key = 0;        // 1 + |x|'s order, 0: no candidate
    int p = INT_MAX;
    double best = 0.0, at_k = 0.0;
#pragma unroll
    for (int m = 0; m < MB; ++m) {
      const int i = 32 * m + lane;
      const long long kx = (i >= k && i < n) ? pivot_key(x[m]) : -1;
      if (kx >= 0 && (unsigned long long)kx + 1 > key) {
        key = (unsigned long long)kx + 1;
        p = i;
        best = x[m];
      }
      if (m == (k >> 5)) at_k = x[m];
    }
    warp_first_max(key, p);
    const double old = __shfl_sync(0xffffffffu, at_k, k & 31);
    const bool found = p != INT_MAX;
    const double akk = __shfl_sync(0xffffffffu, found ? best : at_k, found ? p & 31 : k & 31);
    if (!found) p = k;                 // column of NaNs: keep the row
    const uint32_t hi = (uint32_t)__double2hiint(akk) & 0x7FFFFFFFu;
    const uint32_t lo = (uint32_t)__double2loint(akk);
    const bool nz = (hi | lo) != 0;    // NaN included
    // |akk| >= DBL_MIN (false for NaN)
    const bool use_recip = hi >= 0x00100000u && (hi < 0x7FF00000u || (hi == 0x7FF00000u && lo == 0));
    if (lane == 0) {
      s_p[k & 1] = nz ? p : k;
      gp[k] = p;
    }
    if (nz) {
      const double r = 1.0 / akk;
#pragma unroll
      for (int m = 0; m < MB; ++m) {
        if (32 * m + 31 < k || 32 * m >= n) continue;  // uniform
        const int i = 32 * m + lane;
        if (i == p) x[m] = old;
        if (i > k) x[m] = scale_pivot(x[m], akk, r, use_recip);
        if (i == k) x[m] = akk;
      }
    } else if (my_info == 0) {
      my_info = k + 1;
    }
#pragma unroll
    for (int m = 0; m < MB; ++m) {
      const int i = 32 * m + lane;
      if (i >= k && i < n) A[i * ld + k] = x[m];
    }
  };
  if (warp == 0) {
#pragma unroll
    for (int m = 0; m < MB; ++m) x[m] = (32 * m + lane < n) ? A[(32 * m + lane) * ld] : 0.0;
    pivot(0);
  }
  for (int k = 0; k < n; ++k) {
    __syncthreads();
    const int p = s_p[k & 1];
    if (warp == 0) {
      if (k + 1 < n) {
        const double uk = A[p * ld + k + 1], ok = A[k * ld + k + 1];
#pragma unroll
        for (int m = 0; m < MB; ++m) {
          if (32 * m + 31 <= k || 32 * m >= n) continue;  // uniform
          const int i = 32 * m + lane;
          if (i > k && i < n) x[m] = fma(-x[m], uk, i == p ? ok : A[i * ld + k + 1]);
        }
        __syncwarp();
        if (lane == 0) A[k * ld + k + 1] = uk;
        pivot(k + 1);
      }
    } else {
      if (p != k) {                    // the multipliers of the columns before
        for (int j = tid - 32; j < k; j += (int)blockDim.x - 32) {
          const double t = A[k * ld + j];
          A[k * ld + j] = A[p * ld + j];
          A[p * ld + j] = t;
        }
      }
      small_update_n<2 * MB>((n - k - 2 + 15) >> 4, A, ld, n, k, p, k + 2 * warp - 1,
                             2 * (nwarps - 1), lane, (int)blockDim.x - 32);
    }
  }
  __syncthreads();
  for (int e0 = tid; e0 < n * n; e0 += kLoads * (int)blockDim.x) {
#pragma unroll
    for (int q = 0; q < kLoads; ++q) {
      const int e = e0 + q * (int)blockDim.x;
      if (e < n * n) g[e] = A[(e / n) * ld + e % n];
    }
  }
  if (tid == 0) info[b] = my_info;
}

// ---------------------------------------------------------------------------
// n <= kSmallMax with fewer matrices than SMs: a cluster of two CTAs per
// matrix, so twice as many SMs share the FP64 work.  CTA r of the pair holds
// the columns j = r, r + 2, ... (local column j >> 1, row stride odd) in its
// shared memory.  Step k: the CTA that owns column k searches the pivot,
// swaps rows k and p in its columns, scales column k and writes the
// multipliers l(i) and p into both CTAs' buffers (distributed shared memory);
// after one cluster barrier the other CTA swaps rows in its columns and both
// apply the rank-1 update to their trailing columns.  Every element receives
// the same FMA chain as in getrf_small_kernel, so factors and pivots are
// bit-identical to it (and to getf2).  The l and p buffers alternate with the
// parity of k: the owner of step k + 2 (the same CTA) rewrites them only
// after both CTAs have passed the barrier of step k + 1.
// ---------------------------------------------------------------------------
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kSmallThreads)
getrf_small_pair_kernel(int n, double* __restrict__ a, int64_t stride_a,
                        int32_t* __restrict__ piv, int64_t stride_piv,
                        int32_t* __restrict__ info) {
  namespace cg = cooperative_groups;
  extern __shared__ double smem_lu[];
  __shared__ double s_l[2][kSmallMax];
  __shared__ int s_p[2];
  __shared__ int s_info[2];
  __shared__ int s_pl, s_recip;
  __shared__ double s_akk, s_old, s_rcp;
  cg::cluster_group cluster = cg::this_cluster();
  const int r = (int)cluster.block_rank();
  const int peer = r ^ 1;
  const int ncl = (n + 1 - r) >> 1;          // columns j = r, r + 2, ... < n
  const int ldl = ((n + 1) >> 1) | 1;
  double* A = smem_lu;
  const int tid = threadIdx.x, lane = tid & 31;
  const int tx = tid & 31, ty = tid >> 5;
  const int64_t b = blockIdx.x >> 1;
  double* g = a + b * stride_a;
  int32_t* gp = piv + b * stride_piv;
  double* peer_l = cluster.map_shared_rank(&s_l[0][0], peer);
  int* peer_p = cluster.map_shared_rank(&s_p[0], peer);
  for (int e = tid; e < n * ncl; e += blockDim.x) {
    const int i = e / ncl, jl = e - i * ncl;
    A[i * ldl + jl] = g[(int64_t)i * n + 2 * jl + r];
  }
  int my_info = 0;
  cluster.sync();   // both CTAs run before any remote store
  for (int k = 0; k < n; ++k) {
    const int buf = k & 1;
    if (r == (k & 1)) {
      const int kl = k >> 1;
      if (tid < 32) {
        long long v = -1;
        int idx = INT_MAX;
        for (int i = k + lane; i < n; i += 32) {
          const long long x = pivot_key(A[i * ldl + kl]);
          if (x > v) { v = x; idx = i; }
        }
        warp_argmax_first_key(v, idx);
        if (lane == 0) {
          if (idx == INT_MAX) idx = k;  // column of NaNs: keep the row
          s_pl = idx;
          const double akk = A[idx * ldl + kl];
          s_akk = akk;
          s_old = A[k * ldl + kl];
          s_recip = fabs(akk) >= DBL_MIN;
          s_rcp = 1.0 / akk;
          gp[k] = idx;
        }
      }
      __syncthreads();
      const int p = s_pl;
      const double akk = s_akk;
      if (akk != 0.0) {
        if (p != k) {
          for (int jl = tid; jl < ncl; jl += blockDim.x) {
            if (jl == kl) continue;
            const double t = A[k * ldl + jl];
            A[k * ldl + jl] = A[p * ldl + jl];
            A[p * ldl + jl] = t;
          }
        }
        const bool use_recip = s_recip != 0;
        const double rcp = s_rcp;
        if (tid == 0) A[k * ldl + kl] = akk;
        for (int i = k + 1 + tid; i < n; i += blockDim.x) {
          const double v = (i == p) ? s_old : A[i * ldl + kl];
          const double lv = scale_pivot(v, akk, rcp, use_recip);
          A[i * ldl + kl] = lv;
          s_l[buf][i] = lv;
          peer_l[buf * kSmallMax + i] = lv;
        }
      } else {
        if (my_info == 0) my_info = k + 1;
        for (int i = k + 1 + tid; i < n; i += blockDim.x) {
          const double lv = A[i * ldl + kl];
          s_l[buf][i] = lv;
          peer_l[buf * kSmallMax + i] = lv;
        }
      }
      if (tid == 0) {
        const int pe = (akk != 0.0) ? p : k;   // the row the other CTA swaps with k
        s_p[buf] = pe;
        peer_p[buf] = pe;
      }
    }
    cluster.sync();
    if (r != (k & 1)) {
      const int p = s_p[buf];
      if (p != k) {
        for (int jl = tid; jl < ncl; jl += blockDim.x) {
          const double t = A[k * ldl + jl];
          A[k * ldl + jl] = A[p * ldl + jl];
          A[p * ldl + jl] = t;
        }
        __syncthreads();
      }
    }
    // rank-1 update of this CTA's trailing columns j = 2 jl + r > k
    const int jl0 = (k + 2 - r) >> 1;
    const int nchunk = (ncl - jl0 + 31) >> 5;
    constexpr int kMaxChunk = ((kSmallMax + 1) / 2 + 31) / 32;
    double u[kMaxChunk];
#pragma unroll
    for (int c = 0; c < kMaxChunk; ++c) {
      if (c >= nchunk) break;
      const int jl = jl0 + tx + 32 * c;
      u[c] = (jl < ncl) ? A[k * ldl + jl] : 0.0;
    }
    for (int i = k + 1 + ty; i < n; i += (kSmallThreads >> 5)) {
      const double l = s_l[buf][i];
#pragma unroll
      for (int c = 0; c < kMaxChunk; ++c) {
        if (c >= nchunk) break;
        const int jl = jl0 + tx + 32 * c;
        if (jl < ncl) A[i * ldl + jl] = fma(-l, u[c], A[i * ldl + jl]);
      }
    }
    __syncthreads();
  }
  for (int e = tid; e < n * ncl; e += blockDim.x) {
    const int i = e / ncl, jl = e - i * ncl;
    g[(int64_t)i * n + 2 * jl + r] = A[i * ldl + jl];
  }
  // info = the first zero pivot over both CTAs' steps
  if (tid == 0) *cluster.map_shared_rank(&s_info[r], 0) = my_info;
  cluster.sync();
  if (r == 0 && tid == 0) {
    const int i0 = s_info[0], i1 = s_info[1];
    info[b] = (i0 == 0) ? i1 : (i1 == 0 ? i0 : min(i0, i1));
  }
}

// ---------------------------------------------------------------------------
// Blocked path, one matrix at a time (lda = n).
// ---------------------------------------------------------------------------

// getf2 on the panel columns [j0, j0+nb) over rows [j0, n) by one CTA.
// Row interchanges touch only the panel columns; the other columns receive
// them from laswp_kernel.
__global__ void __launch_bounds__(kPanelThreads)
panel_getf2_kernel(int n, int j0, int nb, double* __restrict__ a, int32_t* __restrict__ piv,
                   int32_t* __restrict__ info) {
  __shared__ long long s_v[32];
  __shared__ int s_i[32];
  __shared__ int s_p, s_recip;
  __shared__ double s_akk, s_old, s_rcp;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int nwarps = blockDim.x >> 5;
  for (int k = j0; k < j0 + nb; ++k) {
    long long v = -1;
    int idx = INT_MAX;
    for (int i = k + tid; i < n; i += blockDim.x) {
      const long long x = pivot_key(a[(int64_t)i * n + k]);
      if (x > v) { v = x; idx = i; }
    }
    warp_argmax_first_key(v, idx);
    if (lane == 0) { s_v[warp] = v; s_i[warp] = idx; }
    __syncthreads();
    if (warp == 0) {
      v = lane < nwarps ? s_v[lane] : -1;
      idx = lane < nwarps ? s_i[lane] : INT_MAX;
      warp_argmax_first_key(v, idx);
      if (lane == 0) {
        if (idx == INT_MAX) idx = k;
        s_p = idx;
        const double akk = a[(int64_t)idx * n + k];
        s_akk = akk;
        s_old = a[(int64_t)k * n + k];
        s_recip = fabs(akk) >= DBL_MIN;
        s_rcp = 1.0 / akk;
        piv[k] = idx;
        if (akk == 0.0 && *info == 0) *info = k + 1;
      }
    }
    __syncthreads();
    const int p = s_p;
    const double akk = s_akk;
    if (akk != 0.0) {
      if (p != k) {
        for (int j = j0 + tid; j < j0 + nb; j += blockDim.x) {
          if (j == k) continue;
          const double t = a[(int64_t)k * n + j];
          a[(int64_t)k * n + j] = a[(int64_t)p * n + j];
          a[(int64_t)p * n + j] = t;
        }
      }
      const bool use_recip = s_recip != 0;
      const double r = s_rcp;
      if (tid == 0) a[(int64_t)k * n + k] = akk;
      for (int i = k + 1 + tid; i < n; i += blockDim.x) {
        const double x = (i == p) ? s_old : a[(int64_t)i * n + k];
        a[(int64_t)i * n + k] = scale_pivot(x, akk, r, use_recip);
      }
    }
    __syncthreads();
    // update the remaining panel columns (k, j0+nb) of rows i > k.
    const int w = j0 + nb - (k + 1);
    if (w > 0) {
      for (int e = tid; e < (n - k - 1) * w; e += blockDim.x) {
        const int i = k + 1 + e / w;
        const int j = k + 1 + e % w;
        a[(int64_t)i * n + j] = fma(-a[(int64_t)i * n + k], a[(int64_t)k * n + j], a[(int64_t)i * n + j]);
      }
    }
    __syncthreads();
  }
}

// ---------------------------------------------------------------------------
// getf2 on the panel columns [j0, j0+nb) over a thread-block cluster.
//
// The one-CTA panel is bound by the FP64 pipe of a single SM (2 FMA per clock
// on GB300: 124 us of arithmetic for a 1000 x 32 panel).  Here the rows are
// split over up to 16 CTAs (R each) and every row lives in the registers of
// TPR threads (thread t of a row holds the columns q * TPR + t), so the
// rank-1 updates run on 16 SMs without touching memory.
// A column costs an exchange over the cluster, and what bounds it is latency
// (measured, cycles: cluster barrier 380, plus 35 for each CTA that a candidate
// is stored to, remote load 350, division 330, FP64 FMA 64 and as much for
// every further warp on the sub-partition).  So per column kk:
//   1. the first maximum of |a| over the CTA by integer reductions (warp, one
//      block barrier, again), its (key, row) stored into every CTA's slots;
//   2. while those stores travel, the columns after kk take the update of step
//      kk - 1 (only column kk took it at once), a warp without rows forms
//      the reciprocal of the CTA's candidate, and the candidate's row and row kk
//      are laid out in this CTA's shared memory;
//   3. one cluster barrier; every warp picks the same winner from local slots;
//      the winning row and its reciprocal are read from the winner's CTA;
//   4. rows swapped, column kk scaled, column kk + 1 updated.
// Slots and staging alternate with the column's parity: a CTA rewrites one
// only after the barrier of the next column, which every CTA reaches after it
// has read it.  Arithmetic and pivot choice are those of panel_getf2_kernel.
// Measured, a 32-column panel on average: n = 1000 50 us (158 us on one CTA),
// n = 2003 60 us (301 us); 1.5 us a column at n = 1000: search 0.35, update
// beside division 0.35, barrier 0.25, winner and its row 0.4, scaling 0.2.
// ---------------------------------------------------------------------------
constexpr int kPcluMax = 16;        // CTAs per cluster
constexpr int kPcluRowThreads = 512;                  // threads that hold rows
constexpr int kPcluThreads = kPcluRowThreads + 32;    // and the warp that divides
// Unused dynamic shared memory that a panel CTA reserves, so that no CTA of
// the trailing update running beside it (17 KB each) shares its SM's FP64 pipe.
constexpr int kPcluReserve = 212 * 1024;
constexpr int kPcluRows = 32;       // aimed rows per CTA (fewer CTAs for short panels)
constexpr int kPcluMaxM = kPcluMax * kPcluRowThreads;  // tallest panel (one thread per row)

struct __align__(16) PanelKey {
  unsigned long long key;
  long long idx;
};

struct PanelSmem {
  PanelKey slot[2][kPcluMax];            // candidates of all CTAs, by parity
  PanelKey cand[2][kPcluThreads / 32];   // this CTA's, by parity and warp
  double cval[2][kPcluThreads / 32];     // and their values
  __align__(16) double mine[2][kNB + 2]; // this CTA's candidate row, then its reciprocal
  __align__(16) double minek[2][kNB + 2];  // row kk (its owner's; no reciprocal)
  __align__(16) double prow[2][kNB + 2]; // the pivot row and reciprocal, received
  __align__(16) double rowk[kNB];        // row kk, received by the pivot row's owner
};

template <int TPR>
__global__ void __launch_bounds__(kPcluThreads, 1)
panel_getf2_cluster_kernel(int n, int j0, int nb, int rows_per_cta, double* __restrict__ a,
                           int32_t* __restrict__ piv, int32_t* __restrict__ info) {
  namespace cg = cooperative_groups;
  constexpr int Q = kNB / TPR;      // columns per thread
  __shared__ PanelSmem sm;
  cg::cluster_group cluster = cg::this_cluster();
  const int ncta = (int)cluster.num_blocks();
  const int rank = (int)cluster.block_rank();
  const int m = n - j0;
  const int R = rows_per_cta;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nwarps = (int)blockDim.x >> 5;
  const int lr = tid / TPR, t = tid % TPR;
  const int gi = rank * R + lr;     // panel row
  const bool has = lr < R && gi < m;
  double r[Q];
  pdl_wait();
  // everything before this panel is finished: the rest of the previous
  // panel's trailing update may start beside it
  pdl_trigger();
#pragma unroll
  for (int q = 0; q < Q; ++q) {
    const int c = q * TPR + t;
    r[q] = (has && c < nb) ? a[(int64_t)(j0 + gi) * n + j0 + c] : 0.0;
  }
  int bad = 0;
  double l = 0.0;                   // this row's multiplier of the step before
  bool act = false;                 // and whether that step updates the row
  cluster.sync();                   // every CTA runs before any remote store
#pragma unroll
  for (int q = 0; q < Q; ++q) {
#pragma unroll 1
    for (int tt = 0; tt < TPR; ++tt) {
      const int kk = q * TPR + tt;
      if (kk >= nb) break;          // uniform over the cluster
      const int par = kk & 1;
      // 1. the CTA's first max |a| in column kk (key 0: none, NaN)
      unsigned long long key = 0;
      int idx = INT_MAX;
      if (has && t == tt && gi >= kk) {
        const long long b = pivot_key(r[q]);
        if (b >= 0) { key = (unsigned long long)b + 1; idx = gi; }
      }
      warp_first_max(key, idx);
      if (lane == 0) { sm.cand[par][warp].key = key; sm.cand[par][warp].idx = idx; }
      if (has && t == tt && gi == idx) sm.cval[par][warp] = r[q];
      __syncthreads();
      key = lane < nwarps ? sm.cand[par][lane].key : 0ull;
      idx = lane < nwarps ? (int)sm.cand[par][lane].idx : INT_MAX;
      const unsigned long long wk = key;
      const int wi = idx;
      warp_first_max(key, idx);
      if (warp == 0 && lane < ncta) {
        PanelKey* dst = cluster.map_shared_rank(&sm.slot[par][rank], lane);
        *reinterpret_cast<longlong2*>(dst) = make_longlong2((long long)key, (long long)idx);
      }
      // 2. meanwhile the rest of step kk - 1, and what the others will read
      if (warp == nwarps - 1) {
        const unsigned mask = __ballot_sync(0xffffffffu, wk == key && wi == idx);
        const double rc = 1.0 / sm.cval[par][__ffs(mask) - 1];
        if (lane == 0) sm.mine[par][kNB] = rc;
      }
      if (act) {
#pragma unroll
        for (int c = q + 1; c < Q; ++c) r[c] = fma(-l, sm.prow[par ^ 1][c * TPR + t], r[c]);
      }
      if (has && gi == idx) {
#pragma unroll
        for (int c = 0; c < Q; ++c) sm.mine[par][c * TPR + t] = r[c];
      }
      if (has && gi == kk) {
#pragma unroll
        for (int c = 0; c < Q; ++c) sm.minek[par][c * TPR + t] = r[c];
      }
      cluster.sync();               // the one cluster barrier of the column
      // 3. the winner, from local shared memory (the same in every CTA)
      key = lane < ncta ? sm.slot[par][lane].key : 0ull;
      idx = lane < ncta ? (int)sm.slot[par][lane].idx : INT_MAX;
      warp_first_max(key, idx);
      const bool none = key == 0ull;          // a column of NaNs: row kk stays
      const int p = none ? kk : idx;
      const int own_p = p / R, own_k = kk / R;
      if (warp == nwarps - 1) {
        if (lane <= kNB / 2) {      // the row and, behind it, the reciprocal
          const double* src = cluster.map_shared_rank(none ? sm.minek[par] : sm.mine[par], own_p);
          reinterpret_cast<double2*>(sm.prow[par])[lane] =
              reinterpret_cast<const double2*>(src)[lane];
        }
      } else if (warp == 0 && own_p == rank) {
        sm.rowk[lane] = cluster.map_shared_rank(sm.minek[par], own_k)[lane];
      }
      __syncthreads();
      const double* prow = sm.prow[par];
      const double akk = prow[kk];
      const bool live = (__double_as_longlong(akk) << 1) != 0;  // akk != 0 (NaN included)
      if (live && p != kk && has) {
        if (gi == kk) {
#pragma unroll
          for (int c = 0; c < Q; ++c) r[c] = prow[c * TPR + t];
        } else if (gi == p) {
#pragma unroll
          for (int c = 0; c < Q; ++c) r[c] = sm.rowk[c * TPR + t];
        }
      }
      if (rank == 0 && tid == 0) {
        piv[j0 + kk] = j0 + p;
        if (!live && bad == 0) bad = j0 + kk + 1;
      }
      // 4. column kk scaled; the update of column kk + 1 (with the rest of
      // its register column), the others follow in the next step
      act = has && gi > kk;
      l = r[q];
      if (live && act && t == tt) {
        // |akk| >= DBL_MIN (false for NaN) from its bits: an FP64 comparison
        // would take the FP64 pipe like a multiplication
        const unsigned hi = (unsigned)__double2hiint(akk) & 0x7FFFFFFFu;
        const bool use_recip = hi - 0x00100000u < 0x7FE00000u ||
                               (hi == 0x7FF00000u && __double2loint(akk) == 0);
        l = scale_pivot(l, akk, prow[kNB], use_recip);
        r[q] = l;
      }
      if (TPR > 1) l = __shfl_sync(0xffffffffu, l, (lane & ~(TPR - 1)) | tt);
      if (tt + 1 < TPR) {
        if (act && t > tt) r[q] = fma(-l, prow[q * TPR + t], r[q]);
      } else if (q + 1 < Q) {
        if (act) r[q + 1 < Q ? q + 1 : q] = fma(-l, prow[(q + 1) * TPR + t], r[q + 1 < Q ? q + 1 : q]);
      }
    }
  }
#pragma unroll
  for (int q = 0; q < Q; ++q) {
    const int c = q * TPR + t;
    if (has && c < nb) a[(int64_t)(j0 + gi) * n + j0 + c] = r[q];
  }
  if (rank == 0 && tid == 0 && bad != 0 && *info == 0) *info = bad;
  cluster.sync();  // no CTA leaves while another may still read its shared memory
}

template <int TPR>
static int launch_panel_clu(int c, int R, int n, int j0, int nb, double* a, int32_t* piv,
                            int32_t* info, cudaStream_t st) {
  if (!cluster_fits(reinterpret_cast<const void*>(panel_getf2_cluster_kernel<TPR>), c, kPcluThreads,
                    kPcluReserve))
    return -1;
  const int threads = (R * TPR + 31) / 32 * 32 + 32;
  const cudaError_t e =
      launch_pdl(panel_getf2_cluster_kernel<TPR>, dim3((unsigned)c), dim3((unsigned)threads),
                 kPcluReserve, st, c, n, j0, nb, R, a, piv, info);
  if (e != cudaSuccess) {
    cudaGetLastError();
    return -1;
  }
  return 0;
}

// 0 when the cluster panel was launched, -1 when the one-CTA panel must do it
// (a panel above kPcluMaxM rows, or no room for the cluster).  Four threads
// per row up to 128 rows per CTA (2048 rows), then two, then one: the FP64
// pipe bounds the update, so what counts is that all four SM sub-partitions
// of a CTA hold warps even when it has only 32 to 64 rows.
static int launch_panel(int n, int j0, int nb, double* a, int32_t* piv, int32_t* info,
                        cudaStream_t st) {
  const int m = n - j0;
  if (m > kPcluMaxM) return -1;
  int c = (m + kPcluRows - 1) / kPcluRows;
  if (c > kPcluMax) c = kPcluMax;
  const int R = (m + c - 1) / c;
  c = (m + R - 1) / R;              // no empty CTA
  if (R <= kPcluRowThreads / 4) return launch_panel_clu<4>(c, R, n, j0, nb, a, piv, info, st);
  if (R <= kPcluRowThreads / 2) return launch_panel_clu<2>(c, R, n, j0, nb, a, piv, info, st);
  return launch_panel_clu<1>(c, R, n, j0, nb, a, piv, info, st);
}

// The panel's row interchanges on the columns outside it, and for the columns
// right of it the block row U12 = L11^{-1} A12 (unit lower, column-oriented
// substitution a(i,j) = fma(-l(i,k), a(k,j), a(i,j)), k ascending).
//
// A CTA takes kStCols columns, one warp per column with lane i holding row
// j0 + i: a step is one shuffle and one FMA per warp, 31 FP64 instructions
// per column that spread over all SMs (one thread per column put the 496
// FMAs of 32 columns on one sub-partition: 34 us per panel at n = 1000).
// The rows the interchanges touch (the panel's 32 and up to 32 others) are
// loaded at once into shared memory, swapped there, and written back.  Per
// panel 8 us at n = 1000 (interchanges 4 + one-thread-per-column TRSM 34 before).
constexpr int kStCols = 8;

__global__ void __launch_bounds__(32 * kStCols)
swap_trsm_kernel(int n, int j0, int nb, double* __restrict__ a, const int32_t* __restrict__ piv) {
  __shared__ double L[kNB][kNB + 1];
  __shared__ double X[2 * kNB][kStCols + 1];
  __shared__ int s_slot[kNB], s_row[2 * kNB];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int left = (j0 + kStCols - 1) / kStCols;         // strips left of the panel
  const bool right = (int)blockIdx.x >= left;
  const int c0 = right ? j0 + nb + ((int)blockIdx.x - left) * kStCols : (int)blockIdx.x * kStCols;
  const int cend = right ? n : j0;
  pdl_wait();
  if (warp == 0) {
    // slot of interchange k's partner: a panel row, or 32 + the first lane
    // that names the same outside row
    const int p = (lane < nb) ? piv[j0 + lane] : j0 + lane;
    const unsigned same = __match_any_sync(0xffffffffu, p);
    const bool inside = p < j0 + kNB;                    // rows past n only pad the block
    const int first = __ffs(same) - 1;
    s_slot[lane] = inside ? p - j0 : kNB + first;
    s_row[lane] = (j0 + lane < n) ? j0 + lane : -1;
    s_row[kNB + lane] = (!inside && first == lane) ? p : -1;
  }
  if (right)
    for (int e = tid; e < kNB * kNB; e += 32 * kStCols) {
      const int i = e / kNB, k = e % kNB;
      L[i][k] = (i < nb && k < i) ? a[(int64_t)(j0 + i) * n + j0 + k] : 0.0;
    }
  __syncthreads();
  for (int e = tid; e < 2 * kNB * kStCols; e += 32 * kStCols) {
    const int i = e / kStCols, c = e % kStCols;
    const int row = s_row[i];
    if (row >= 0 && c0 + c < cend) X[i][c] = a[(int64_t)row * n + c0 + c];
  }
  __syncthreads();
  if (tid < kStCols) {
#pragma unroll 4
    for (int k = 0; k < nb; ++k) {
      const int s = s_slot[k];
      const double u = X[k][tid], v = X[s][tid];
      X[k][tid] = v;
      X[s][tid] = u;
    }
  }
  __syncthreads();
  if (right) {
    double x = X[lane][warp];
#pragma unroll
    for (int k = 0; k < kNB - 1; ++k) {
      const double xk = __shfl_sync(0xffffffffu, x, k);
      if (lane > k) x = fma(-L[lane][k], xk, x);
    }
    X[lane][warp] = x;
    __syncthreads();
  }
  pdl_trigger();
  for (int e = tid; e < 2 * kNB * kStCols; e += 32 * kStCols) {
    const int i = e / kStCols, c = e % kStCols;
    const int row = s_row[i];
    if (row >= 0 && c0 + c < cend) a[(int64_t)row * n + c0 + c] = X[i][c];
  }
}

// Trailing update A22 -= L21 U12 (k = j0..j0+nb-1), each element an FMA chain
// from its stored value, on the columns from c_lo on (c_lo a multiple of kGT
// past the panel).  32x32 tile per CTA, 2x4 per thread: the FP64 pipe bounds
// it at any tile size, so small tiles only shorten the last wave (n = 1000: 27
// us a panel against 45 us with 64x64 tiles; n = 2003: 79 against 95).
//
// This is the part of the update that the next panel does not need: it is
// launched behind that panel (a dependent launch, released as soon as the
// panel's CTAs have started) and runs beside it.  It therefore reads at once
// what kernels finished before the panel wrote (through L2: __ldcg), touches
// none of the panel's columns, and waits for the panel only before it ends, so
// that whatever follows it follows both.
constexpr int kGT = 32;
__global__ void __launch_bounds__(128)
gemm_trailing_kernel(int n, int j0, int nb, int c_lo, double* a) {
  __shared__ double Ls[kGT][kNB + 1];
  __shared__ double Us[kNB][kGT + 2];
  const int i0 = j0 + nb + blockIdx.y * kGT;
  const int c0 = c_lo + blockIdx.x * kGT;
  const int tid = threadIdx.x;
  const int tx = tid & 7, ty = tid >> 3;
  double acc[2][4];
#pragma unroll
  for (int r = 0; r < 2; ++r)
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      const int i = i0 + ty + 16 * r, j = c0 + tx + 8 * c;
      acc[r][c] = (i < n && j < n) ? __ldcg(a + (int64_t)i * n + j) : 0.0;
    }
#pragma unroll
  for (int e0 = 0; e0 < kGT * kNB; e0 += 128) {
    const int e = e0 + tid;
    const int r = e / kNB, k = e % kNB;
    Ls[r][k] = (i0 + r < n && k < nb) ? __ldcg(a + (int64_t)(i0 + r) * n + j0 + k) : 0.0;
    Us[r][k] = (c0 + k < n && r < nb) ? __ldcg(a + (int64_t)(j0 + r) * n + c0 + k) : 0.0;
  }
  __syncthreads();
#pragma unroll 8
  for (int k = 0; k < nb; ++k) {
    double l[2], u[4];
#pragma unroll
    for (int r = 0; r < 2; ++r) l[r] = Ls[ty + 16 * r][k];
#pragma unroll
    for (int c = 0; c < 4; ++c) u[c] = Us[k][tx + 8 * c];
#pragma unroll
    for (int r = 0; r < 2; ++r)
#pragma unroll
      for (int c = 0; c < 4; ++c) acc[r][c] = fma(-l[r], u[c], acc[r][c]);
  }
#pragma unroll
  for (int r = 0; r < 2; ++r)
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      const int i = i0 + ty + 16 * r, j = c0 + tx + 8 * c;
      if (i < n && j < n) a[(int64_t)i * n + j] = acc[r][c];
    }
  pdl_wait();
}

// The same update on the next panel's columns [j0+nb, j0+nb+32), ahead of the
// rest.  8x32 tile per CTA: these few columns are on the critical path, and
// only as many SMs work on them as there are tiles.
constexpr int kNxRows = 8;
__global__ void __launch_bounds__(128)
gemm_next_panel_kernel(int n, int j0, int nb, double* __restrict__ a) {
  __shared__ double Ls[kNxRows][kNB + 1];
  __shared__ double Us[kNB][kNB];
  const int s = j0 + nb;
  const int i0 = s + (int)blockIdx.x * kNxRows;
  const int tid = threadIdx.x;
  const int tx = tid & 15, ty = tid >> 4;
  const int i = i0 + ty;
  pdl_wait();
  double acc[2];
#pragma unroll
  for (int c = 0; c < 2; ++c) {
    const int j = s + tx + 16 * c;
    acc[c] = (i < n && j < n) ? a[(int64_t)i * n + j] : 0.0;
  }
#pragma unroll
  for (int e = tid; e < kNxRows * kNB; e += 128) {
    const int r = e / kNB, k = e % kNB;
    Ls[r][k] = (i0 + r < n && k < nb) ? a[(int64_t)(i0 + r) * n + j0 + k] : 0.0;
  }
#pragma unroll
  for (int e = tid; e < kNB * kNB; e += 128) {
    const int k = e / kNB, c = e % kNB;
    Us[k][c] = (s + c < n && k < nb) ? a[(int64_t)(j0 + k) * n + s + c] : 0.0;
  }
  __syncthreads();
#pragma unroll 8
  for (int k = 0; k < nb; ++k) {
    const double l = Ls[ty][k];
#pragma unroll
    for (int c = 0; c < 2; ++c) acc[c] = fma(-l, Us[k][tx + 16 * c], acc[c]);
  }
  pdl_trigger();
#pragma unroll
  for (int c = 0; c < 2; ++c) {
    const int j = s + tx + 16 * c;
    if (i < n && j < n) a[(int64_t)i * n + j] = acc[c];
  }
}

__global__ void zero_info_kernel(int32_t* info, int64_t count) {
  int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i < count) info[i] = 0;
}

// Per panel: its interchanges and block row, the update of the next panel's
// columns, the next panel, and beside that panel the rest of the update.
int getrf_blocked(int n, double* a, int32_t* piv, int32_t* info, cudaStream_t st) {
  zero_info_kernel<<<1, 32, 0, st>>>(info, 1);
  auto panel = [&](int j0) {
    const int nb = min(kNB, n - j0);
    if (launch_panel(n, j0, nb, a, piv, info, st) != 0)
      panel_getf2_kernel<<<1, kPanelThreads, 0, st>>>(n, j0, nb, a, piv, info);
  };
  panel(0);
  for (int j0 = 0; j0 < n; j0 += kNB) {
    const int nb = min(kNB, n - j0);
    const int rest = n - j0 - nb;
    const int strips = (j0 + kStCols - 1) / kStCols + (rest + kStCols - 1) / kStCols;
    if (strips > 0)
      LXGB_CUDA_TRY(launch_pdl(swap_trsm_kernel, dim3((unsigned)strips), dim3(32 * kStCols), 0, st,
                               1, n, j0, nb, a, piv),
                    "getrf: swap_trsm launch");
    if (rest > 0) {
      LXGB_CUDA_TRY(launch_pdl(gemm_next_panel_kernel,
                               dim3((unsigned)((rest + kNxRows - 1) / kNxRows)), dim3(128), 0, st,
                               1, n, j0, nb, a),
                    "getrf: next panel update launch");
      panel(j0 + nb);
      const int wide = rest - kNB;               // columns after the next panel's
      if (wide > 0)
        LXGB_CUDA_TRY(launch_pdl(gemm_trailing_kernel,
                                 dim3((unsigned)((wide + kGT - 1) / kGT),
                                      (unsigned)((rest + kGT - 1) / kGT)),
                                 dim3(128), 0, st, 1, n, j0, nb, j0 + nb + kNB, a),
                      "getrf: trailing update launch");
    }
  }
  return check_launch("getrf blocked");
}

// ---------------------------------------------------------------------------
// getrs for n > kSmallMax: the row interchanges as one gather or scatter per
// vector, then two multi-CTA triangular solves (trisolve.cu).
// ---------------------------------------------------------------------------
constexpr int kPermThreads = 1024;
constexpr int kPermRows = 19;                      // values per thread, in registers
constexpr int kPermFew = 4;                        // and up to 4096 rows
constexpr int kPermMaxN = 19200;                   // 12 bytes of shared memory per row
static_assert(kPermMaxN <= kPermRows * kPermThreads, "a register per value");

// x = P x (or Pᵀ x), one CTA per vector: every value is read before the first is written.
template <int ROWS>
__global__ void __launch_bounds__(kPermThreads)
getrs_perm_kernel(int n, const int32_t* __restrict__ piv, int64_t stride_piv,
                  double* __restrict__ b, int64_t stride_b, int trans) {
  extern __shared__ int smem_swaps[];
  int *head = smem_swaps, *next = head + n, *root = next + n;
  const int32_t* p = piv + (int64_t)blockIdx.y * stride_piv;
  double* g = b + (int64_t)blockIdx.y * stride_b + (int64_t)blockIdx.x * n;
  const SwapMode mode = swap_build(n, p, head, next, root, trans != 0);
  const bool scatter = trans && mode != kSwapInOrder;
  double v[ROWS];
#pragma unroll
  for (int u = 0; u < ROWS; ++u) {
    const int i = threadIdx.x + u * (int)blockDim.x;
    if (u * (int)blockDim.x >= n) break;           // uniform
    v[u] = i < n ? g[scatter ? i : swap_source(mode, i, p, head, next, root)] : 0.0;
  }
  __syncthreads();
#pragma unroll
  for (int u = 0; u < ROWS; ++u) {
    const int i = threadIdx.x + u * (int)blockDim.x;
    if (u * (int)blockDim.x >= n) break;
    if (i < n) g[scatter ? swap_source(mode, i, p, head, next, root) : i] = v[u];
  }
}

// The same, in order and in global memory, for n above kPermMaxN.
__global__ void getrs_swap_kernel(int n, const int32_t* __restrict__ piv, int64_t stride_piv,
                                  double* __restrict__ b, int64_t stride_b, int trans) {
  const int32_t* p = piv + (int64_t)blockIdx.y * stride_piv;
  double* x = b + (int64_t)blockIdx.y * stride_b + (int64_t)blockIdx.x * n;
  for (int s = 0; s < n; ++s) {
    const int k = trans ? n - 1 - s : s;
    const int q = p[k];
    if (q != k) { const double v = x[k]; x[k] = x[q]; x[q] = v; }
  }
}

static int getrs_perm(int64_t batch, int n, int nrhs, const int32_t* piv, int64_t stride_piv,
                      double* b, int64_t stride_b, int trans, cudaStream_t st) {
  const dim3 grid((unsigned)nrhs, (unsigned)batch);
  if (n > kPermMaxN) {
    getrs_swap_kernel<<<grid, 1, 0, st>>>(n, piv, stride_piv, b, stride_b, trans);
    return check_launch("getrs swap");
  }
  const size_t smem = (size_t)n * 3 * sizeof(int);
  auto fn = n <= kPermFew * kPermThreads ? getrs_perm_kernel<kPermFew> : getrs_perm_kernel<kPermRows>;
  LXGB_CUDA_TRY(ensure_dynamic_smem(reinterpret_cast<const void*>(fn), (int)smem),
                "getrs: set smem");
  const int threads = n < kPermThreads ? (n + 31) / 32 * 32 : kPermThreads;
  fn<<<grid, threads, smem, st>>>(n, piv, stride_piv, b, stride_b, trans);
  return check_launch("getrs perm");
}

// ---------------------------------------------------------------------------
// getrs for n <= kSmallMax: one CTA per system, the factors staged in shared
// memory, one warp per right-hand side and 32 unknowns (lane l of warp m owns
// row 32 m + l).  A sweep goes by half blocks of 16 unknowns: their warp
// substitutes (a shuffle and an FMA per unknown; with U also x_t * (1 / u_tt),
// within one rounding of the quotient, the inverses formed up front), then the
// other warps subtract them from their rows while it goes on with its second
// half.  The dependent chain of a step is what bounds it: one warp with all the
// rows of a right-hand side issues its FMAs for every 32 rows one after the
// other on GB300's narrow FP64 pipe.  Interchanges: every thread follows one
// element through the n swaps, all in parallel.
// Measured (one right-hand side): 16.6 us at n = 48, 37 at 128, 53 at 168, against
// 29, 72 and 98 with one warp per right-hand side.
// ---------------------------------------------------------------------------
constexpr int kSmallRhs = 4;           // groups of right-hand sides at a time
constexpr int kSmallSolveThreads = 32 * kSmallBlocks * kSmallRhs;
constexpr int kSmallHalf = 16;

// One sweep over op(T), ascending (FWD) or descending, on the x of this thread
// (row 32 m + lane of NV right-hand sides, rinv the inverse of its diagonal);
// op(T)[i][t] is T[t][i] with TR.  xs: the unknowns of two half blocks in turn, by
// right-hand side.
template <bool FWD, bool UNIT, bool TR, int NV>
__device__ __forceinline__ void small_sweep(int n, int ld, const double* T, double rinv,
                                            double* xs, int nblk, int m, int lane, bool active,
                                            double (&x)[NV]) {
  constexpr int kH = kSmallHalf;
  const int i = 32 * m + lane;
  for (int q = 0; q < 2 * nblk; ++q) {
    const int hb = FWD ? q : 2 * nblk - 1 - q;      // half block: unknowns 16 hb ..
    const int t0 = kH * hb;
    if (active && m == (hb >> 1)) {
      double tv[kH];
#pragma unroll
      for (int u = 0; u < kH; ++u) {
        const int t = FWD ? t0 + u : t0 + kH - 1 - u;
        const bool use = t < n && i < n && (FWD ? i > t : i < t);
        tv[u] = use ? (TR ? T[t * ld + i] : T[i * ld + t]) : 0.0;
      }
#pragma unroll
      for (int u = 0; u < kH; ++u) {
        const int t = FWD ? t0 + u : t0 + kH - 1 - u;
        if (t < n) {
          double xt[NV];
#pragma unroll
          for (int v = 0; v < NV; ++v) {
            if (!UNIT && i == t) x[v] *= rinv;
            xt[v] = __shfl_sync(0xffffffffu, x[v], t & 31);
          }
#pragma unroll
          for (int v = 0; v < NV; ++v)
            if (i < n && (FWD ? i > t : i < t)) x[v] = fma(-tv[u], xt[v], x[v]);
        }
      }
      if ((i >> 4) == hb) {
#pragma unroll
        for (int v = 0; v < NV; ++v) xs[2 * kH * v + kH * (q & 1) + (i & (kH - 1))] = x[v];
      }
    }
    __syncthreads();
    if (active && i < n && (FWD ? m > (hb >> 1) : m < (hb >> 1))) {
      double tv[kH];
#pragma unroll
      for (int u = 0; u < kH; ++u) {
        const int t = FWD ? t0 + u : t0 + kH - 1 - u;
        tv[u] = t < n ? (TR ? T[t * ld + i] : T[i * ld + t]) : 0.0;
      }
#pragma unroll
      for (int u = 0; u < kH; ++u) {
        const int t = FWD ? t0 + u : t0 + kH - 1 - u;
        if (t < n) {
#pragma unroll
          for (int v = 0; v < NV; ++v)
            x[v] = fma(-tv[u], xs[2 * kH * v + kH * (q & 1) + (t & (kH - 1))], x[v]);
        }
      }
    }
  }
}

template <int NV>
__global__ void __launch_bounds__(kSmallSolveThreads)
getrs_small_kernel(int n, int nrhs, int per, const double* __restrict__ lu, int64_t stride_a,
                   const int32_t* __restrict__ piv, int64_t stride_piv, double* __restrict__ b,
                   int64_t stride_b, int trans) {
  extern __shared__ double smem_x[];
  const int ld = n | 1;
  const int nblk = (n + 31) >> 5;
  double* T = smem_x;                                   // n × ld
  double* rinv = T + (int64_t)n * ld;                   // 1 / u_tt
  double* xs = rinv + n;                                // finished unknowns, by right-hand side
  int* perm = reinterpret_cast<int*>(xs + per * NV * 2 * kSmallHalf);  // x_perm[i] = b[perm[i]]
  int* sp = perm + n;                                   // the interchanges
  const int sys = blockIdx.x;
  const double* A = lu + (int64_t)sys * stride_a;
  const int32_t* P = piv + (int64_t)sys * stride_piv;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  for (int i = tid; i < n; i += blockDim.x) sp[i] = P[i];
  constexpr int kLoads = 8;
  for (int e0 = tid; e0 < n * n; e0 += kLoads * blockDim.x) {
    double v[kLoads];
#pragma unroll
    for (int u = 0; u < kLoads; ++u) {
      const int e = e0 + u * (int)blockDim.x;
      v[u] = e < n * n ? A[e] : 0.0;
    }
#pragma unroll
    for (int u = 0; u < kLoads; ++u) {
      const int e = e0 + u * (int)blockDim.x;
      if (e < n * n) T[(e / n) * ld + e % n] = v[u];
    }
  }
  __syncthreads();
  for (int i = tid; i < n; i += blockDim.x) {
    int pos = i;                       // where element i is after the swaps
#pragma unroll 8
    for (int k = 0; k < n; ++k) {
      const int p = sp[k];
      pos = pos == k ? p : (pos == p ? k : pos);
    }
    perm[pos] = i;
    rinv[i] = 1.0 / T[i * ld + i];
  }
  __syncthreads();
  const int rg = warp / nblk, m = warp - rg * nblk, i = 32 * m + lane;
  const double ri = i < n ? rinv[i] : 0.0;
  for (int r0 = 0; r0 < nrhs; r0 += per * NV) {
    const int first = r0 + rg * NV;                      // this warp's right-hand sides
    const bool active = rg < per && first < nrhs;
    double* g = b + (int64_t)sys * stride_b + (int64_t)first * n;
    double* mine = xs + (active ? rg : 0) * NV * 2 * kSmallHalf;
    double x[NV];
#pragma unroll
    for (int v = 0; v < NV; ++v)
      x[v] = (active && i < n && first + v < nrhs) ? g[v * n + (trans ? i : perm[i])] : 0.0;
    // every element is read before the first is written
    __syncthreads();
    if (!trans) {
      small_sweep<true, true, false, NV>(n, ld, T, ri, mine, nblk, m, lane, active, x);   // L y = P b
      small_sweep<false, false, false, NV>(n, ld, T, ri, mine, nblk, m, lane, active, x); // U x = y
    } else {
      small_sweep<true, false, true, NV>(n, ld, T, ri, mine, nblk, m, lane, active, x);   // Uᵀ z = b
      small_sweep<false, true, true, NV>(n, ld, T, ri, mine, nblk, m, lane, active, x);   // Lᵀ w = z
    }
#pragma unroll
    for (int v = 0; v < NV; ++v)                         // x = Pᵀ w: x[perm[i]] = w[i]
      if (active && i < n && first + v < nrhs) g[v * n + (trans ? perm[i] : i)] = x[v];
  }
}

}  // namespace lxgb

using namespace lxgb;

// 1: batches of at most half the SM count with n in [32, 168] run on two-CTA
// clusters; 0 (the default): one CTA per matrix.  The pair halves each SM's
// FP64 work but adds a cluster barrier and a distributed-shared-memory
// exchange to every column; on the 64 × n = 128 batch it factors in 0.44 ms
// against 0.33 ms for one CTA with the lookahead pivot search.
static int g_getrf_pair = 0;

extern "C" int lxgb_getrf_set_pair(int32_t on) {
  g_getrf_pair = on ? 1 : 0;
  return LXGB_SUCCESSFUL;
}

extern "C" int lxgb_getrf_batched_f64(int64_t batch, int32_t n, double* a, int64_t stride_a,
                                      int32_t* piv, int64_t stride_piv, int32_t* info,
                                      void* stream) {
  LXGB_REQUIRE(batch >= 0 && n >= 0, "getrf: batch and n must be non-negative");
  if (batch == 0 || n == 0) return LXGB_SUCCESSFUL;
  LXGB_REQUIRE(a && piv && info, "getrf: null pointer");
  LXGB_REQUIRE(stride_a >= (int64_t)n * n && stride_piv >= n, "getrf: stride too small");
  cudaStream_t st = as_stream(stream);
  if (n <= kSmallMax && n >= 32 && 2 * batch <= sm_count() && g_getrf_pair) {
    // fewer matrices than SMs: two CTAs (a cluster) per matrix
    const size_t smem = (size_t)n * (((n + 1) >> 1) | 1) * sizeof(double);
    LXGB_CUDA_TRY(ensure_dynamic_smem(reinterpret_cast<const void*>(getrf_small_pair_kernel),
                                      (int)smem),
                  "getrf pair: set smem");
    getrf_small_pair_kernel<<<(unsigned)(2 * batch), kSmallThreads, smem, st>>>(
        n, a, stride_a, piv, stride_piv, info);
    return check_launch("getrf small pair");
  }
  if (n <= kSmallMax) {
    const size_t smem = (size_t)n * (n | 1) * sizeof(double);
    // More warps where the update is the longer part: us per matrix with 256 and
    // 512 threads 14.6 and 16.6 at n = 16, 47 and 47 at 48, 191 and 176 at 100, 317
    // and 289 at 128; 512 matrices of order 64 156 and 187.  Fewer where the shared
    // memory of an SM holds several matrices and there is more than one for each SM: a
    // CTA of 512 threads takes more than half of an SM's registers.  us for 4096 matrices with
    // 128, 256 and 512 threads: n = 65 1067, 1209 and 2278, 80 1850, 1856 and 3071, 96
    // 3124, 2812 and 4240, 119 7206, 5391 and 6746; for 304: n = 65 141, 124 and 185.
    const bool several = batch > sm_count() && 2 * (smem + 2048) <= kSmSharedBytes;
    const int threads = n <= 64 ? kSmallThreads
                                : (!several ? kSmallMaxThreads
                                            : (n <= 80 && batch > 2 * sm_count() ? kSmallThreads / 2
                                                                                 : kSmallThreads));
    // registers for the rows of a column per lane of warp 0
    auto fn = n <= 64 ? getrf_small_kernel<2>
                      : (n <= 128 ? getrf_small_kernel<4> : getrf_small_kernel<kSmallBlocks>);
    LXGB_CUDA_TRY(ensure_dynamic_smem(reinterpret_cast<const void*>(fn), (int)smem),
                  "getrf: set smem");
    for (int64_t off = 0; off < batch; off += 65535LL * 1024) {
      const int64_t cnt = (batch - off < 65535LL * 1024) ? batch - off : 65535LL * 1024;
      fn<<<(unsigned)cnt, threads, smem, st>>>(
          n, a + off * stride_a, stride_a, piv + off * stride_piv, stride_piv, info + off);
    }
    return check_launch("getrf small");
  }
  for (int64_t s = 0; s < batch; ++s) {
    int rc = getrf_blocked(n, a + s * stride_a, piv + s * stride_piv, info + s, st);
    if (rc) return rc;
  }
  return LXGB_SUCCESSFUL;
}

extern "C" int lxgb_getrs_batched_f64(int64_t batch, int32_t n, int32_t nrhs, const double* lu,
                                      int64_t stride_a, const int32_t* piv, int64_t stride_piv,
                                      double* b, int64_t stride_b, int32_t trans, void* stream) {
  LXGB_REQUIRE(batch >= 0 && n >= 0 && nrhs >= 0, "getrs: negative size");
  if (batch == 0 || n == 0 || nrhs == 0) return LXGB_SUCCESSFUL;
  LXGB_REQUIRE(lu && piv && b, "getrs: null pointer");
  LXGB_REQUIRE(trans == 0 || trans == 1, "getrs: trans must be 0 or 1");
  LXGB_REQUIRE(stride_a >= (int64_t)n * n && stride_piv >= n && stride_b >= (int64_t)n * nrhs,
               "getrs: stride too small");
  LXGB_REQUIRE(batch * (int64_t)nrhs < (1LL << 31), "getrs: too many vectors in one call");
  if (n <= kSmallMax && batch < (1LL << 31)) {
    // Two right-hand sides per warp above four: their chains run side by side (us for 16
    // with one and two: n = 128 149 and 141, 168 246 and 239).  Small orders have little
    // to load, so threads that no right-hand side needs only cost CTAs per SM (us for
    // 4096 systems of one, with 8, 4 and 2 warps: n = 16 57, 39 and 33, 64 161, 123 and
    // 147, 96 267, 310 and 345).
    const int nv = nrhs > kSmallRhs ? 2 : 1;
    const int groups = (nrhs + nv - 1) / nv;
    const int per = groups < kSmallRhs ? groups : kSmallRhs;
    const size_t smem = (size_t)n * (n | 1) * sizeof(double) + (size_t)n * sizeof(double) +
                        (size_t)per * nv * 2 * kSmallHalf * sizeof(double) +
                        (size_t)n * 2 * sizeof(int32_t);
    const int warps = (n + 31) / 32 * per, least = n <= 32 ? 2 : (n <= 64 ? 4 : 8);
    const int threads = 32 * (warps < least ? least : warps);
    auto fn = nv == 2 ? getrs_small_kernel<2> : getrs_small_kernel<1>;
    LXGB_CUDA_TRY(ensure_dynamic_smem(reinterpret_cast<const void*>(fn), (int)smem),
                  "getrs small: set smem");
    fn<<<(unsigned)batch, threads, smem, as_stream(stream)>>>(
        n, nrhs, per, lu, stride_a, piv, stride_piv, b, stride_b, trans);
    return check_launch("getrs small");
  }
  cudaStream_t st = as_stream(stream);
  constexpr int64_t kMaxGrid = 65535;               // vectors and systems per launch
  for (int64_t s0 = 0; s0 < batch; s0 += kMaxGrid) {
    const int64_t sb = batch - s0 < kMaxGrid ? batch - s0 : kMaxGrid;
    for (int64_t r0 = 0; r0 < nrhs; r0 += kMaxGrid) {
      const int kb = (int)(nrhs - r0 < kMaxGrid ? nrhs - r0 : kMaxGrid);
      const double* t = lu + s0 * stride_a;
      const int32_t* p = piv + s0 * stride_piv;
      double* x = b + s0 * stride_b + r0 * n;
      int rc = trans ? LXGB_SUCCESSFUL : getrs_perm(sb, n, kb, p, stride_piv, x, stride_b, 0, st);
      if (!rc)  // L y = P b, or Uᵀ z = b
        rc = trisolve_blocked(sb, n, kb, t, n, stride_a, !trans, trans, !trans, x, stride_b, st);
      if (!rc)  // U x = y, or Lᵀ w = z
        rc = trisolve_blocked(sb, n, kb, t, n, stride_a, trans, trans, trans, x, stride_b, st);
      if (!rc && trans) rc = getrs_perm(sb, n, kb, p, stride_piv, x, stride_b, 1, st);
      if (rc) return rc;
    }
  }
  return LXGB_SUCCESSFUL;
}
