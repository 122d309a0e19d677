// GMRES-IR building blocks for the FP32 LU (lu32.cu):
//
//   lxgb_lu32_inverse — L^{-1} and U^{-1} of the FP32 factor as dense FP32
//     triangles, by blocked substitution against the identity: 64-row
//     diagonal-block solves on the CUDA cores and the off-diagonal updates on
//     the tcgen05 tensor cores (TF32 or 3xTF32, as the factor was made).
//     M = U^{-1} L^{-1} P is then applied with two triangular matrix-vector
//     products that every SM shares, instead of two sequential substitutions.
//   lxgb_lu32_apply — y = U^{-1} (L^{-1} (P x)) for a block of FP64 vectors,
//     in FP32 or in double-float arithmetic (FP64-accurate on the FP32 pipe).
//   lxgb_gemv_df — y = A x or y = b - A x with A held as an FP32 hi + lo pair
//     (48 significant bits), in double-float arithmetic: the FP64 operator
//     product and residual of the refinement at a fraction of the FP64-pipe
//     cost.
//
// Sums are formed in a fixed order: results are bitwise reproducible.
#include <cooperative_groups.h>
#include <cuda_bf16.h>

#include "common.cuh"
#include "df.cuh"
#include "swaps.cuh"
#include "tc_gemm.cuh"

namespace lxgb {

namespace cg = cooperative_groups;

constexpr int kInvNB = 64;     // diagonal block size of the inversion
constexpr int kGvRows = 16;    // rows per CTA of the products
constexpr int kGvRhs = 16;     // right-hand sides per CTA of the products
constexpr int kPermMaxN = 25600;
constexpr int kPermRows = 25;  // rows per thread of the 1024 at kPermMaxN

// (P b)_i = b[perm[i]]: the getrf row interchanges composed into one gather
// (swaps.cuh).  The third array of the walk lives in the output until every row's source
// is known.  One thread running the n dependent exchanges took 327 us at n = 8192.
__global__ void __launch_bounds__(1024)
perm_from_swaps_kernel(int n, const int32_t* __restrict__ piv, int32_t* perm) {
  extern __shared__ int32_t sp[];
  const SwapMode mode = swap_build(n, piv, sp, sp + n, perm, false);
  int src[kPermRows];
#pragma unroll
  for (int u = 0; u < kPermRows; ++u) {
    const int i = threadIdx.x + u * (int)blockDim.x;
    src[u] = i < n ? swap_source(mode, i, piv, sp, sp + n, perm) : 0;
  }
  __syncthreads();
#pragma unroll
  for (int u = 0; u < kPermRows; ++u) {
    const int i = threadIdx.x + u * (int)blockDim.x;
    if (i < n) perm[i] = src[u];
  }
}

__global__ void set_identity_f32_kernel(int n, float* __restrict__ w) {
  for (int r = blockIdx.x; r < n; r += gridDim.x)
    for (int c = threadIdx.x; c < n; c += blockDim.x) w[(int64_t)r * n + c] = (r == c) ? 1.0f : 0.0f;
}

// One block row of the LU or of a triangular inversion, everything between the
// panel (or the previous update) and the tensor-core update in one launch:
//  * strips of 64 columns: the panel's row interchanges (KIND 0), then
//    X = T_jj^{-1} W_j on rows [j0, j0+nb) of w — T_jj the unit-lower (KIND 0,
//    1) or upper (KIND 2) diagonal block of the factor, one column per thread in
//    registers — written back in place and, transposed (64 entries per column,
//    zero padded), as the K-major operand of the update: FP32 (PREC 0), its
//    TF32-exact hi and lo parts (PREC 1) or BF16 (PREC 2).  KIND 0 also has
//    strips left of the panel, which only take the interchanges;
//  * further CTAs: the other operand (the panel's columns, na rows of `a_src`)
//    split or converted the same way (PREC 1 and 2), 64 rows each.
// The rows that the interchanges touch (the panel's 64 and up to 64 others) are
// loaded at once into shared memory and swapped there.  Bound by latency: two
// waits for device memory, 64 dependent swaps and 64 dependent substitution
// steps.  Measured per panel at n = 8192: 15 us (LU), 10 and 19 (lower and upper
// inversion, the latter with 64 divisions in its chain); as separate launches —
// one thread per column swapping in global memory, the substitution, two splits
// — 37 + 19 + 8 (LU) and 19 + 8 (inversions).
constexpr int kBrCols = 64;
constexpr int kBrThreads = 128;
constexpr int kBrT = 16;
constexpr int kBrLoads = kInvNB * kInvNB / kBrThreads;
constexpr int kBrLd = kBrCols + 1;

struct BlockRowArgs {
  int n, j0, nb;
  const float* lu;      // holds T_jj at (j0, j0)
  float* w;             // target matrix (row stride n)
  const int32_t* piv;   // KIND 0
  int c_begin, c_end;   // columns solved
  int strips, left;     // strips in all; of these left of the panel (KIND 0)
  void *b0, *b1;        // operand from X: FP32 / hi, lo / BF16
  const float* a_src;   // the other operand, row stride n
  int na;
  void *a0, *a1;
};

template <int PREC>
__device__ __forceinline__ void br_store(void* p0, void* p1, int64_t at, float v) {
  if (PREC == 0) {
    reinterpret_cast<float*>(p0)[at] = v;
  } else if (PREC == 1) {
    const float h = __uint_as_float(__float_as_uint(v) & 0xFFFFE000u);
    reinterpret_cast<float*>(p0)[at] = h;
    reinterpret_cast<float*>(p1)[at] = v - h;
  } else {
    reinterpret_cast<__nv_bfloat16*>(p0)[at] = __float2bfloat16_rn(v);
  }
}

template <int KIND, int PREC>
__global__ void __launch_bounds__(kBrThreads)
block_row_kernel(BlockRowArgs g) {
  constexpr int kRows = KIND == 0 ? 2 * kInvNB : kInvNB;
  // Tt[k][i] = T[i][k]: for a fixed k the multipliers of all rows i are
  // contiguous (16-byte broadcast loads).  Padding rows/columns past nb hold the
  // identity, so the fully unrolled substitution needs no bounds.
  extern __shared__ __align__(16) float br_smem[];
  float (*Tt)[kInvNB + 4] = reinterpret_cast<float (*)[kInvNB + 4]>(br_smem);
  float (*X)[kBrLd] = reinterpret_cast<float (*)[kBrLd]>(br_smem + kInvNB * (kInvNB + 4));
  __shared__ int s_piv[kInvNB], s_slot[kInvNB], s_row[kRows];
  const int tid = threadIdx.x;
  const int n = g.n, j0 = g.j0, nb = g.nb;
  pdl_wait();
  pdl_trigger();  // a product that needs nothing of this row may start beside it
  if ((int)blockIdx.x >= g.strips) {               // the other operand
    if (PREC != 0) {
      const int r0 = ((int)blockIdx.x - g.strips) * kInvNB;
      float v[kBrLoads];
#pragma unroll
      for (int u = 0; u < kBrLoads; ++u) {
        const int e = tid + u * kBrThreads, r = r0 + e / kInvNB, c = e % kInvNB;
        v[u] = (r < g.na && c < nb) ? __ldcg(g.a_src + (int64_t)r * n + c) : 0.0f;
      }
#pragma unroll
      for (int u = 0; u < kBrLoads; ++u) {
        const int e = tid + u * kBrThreads, r = r0 + e / kInvNB, c = e % kInvNB;
        if (r < g.na) br_store<PREC>(g.a0, g.a1, (int64_t)r * kInvNB + c, v[u]);
      }
    }
    return;
  }
  const bool solve = KIND != 0 || (int)blockIdx.x >= g.left;
  float t[kBrLoads];
  const int c0 = solve ? g.c_begin + ((int)blockIdx.x - (KIND == 0 ? g.left : 0)) * kBrCols
                       : (int)blockIdx.x * kBrCols;
  const int cend = solve ? g.c_end : j0;
  if (KIND == 0) {
    if (tid < kInvNB) s_piv[tid] = (tid < nb) ? g.piv[j0 + tid] : j0 + tid;
    __syncthreads();
    if (tid < kInvNB) {
      // slot of interchange k's partner: a panel row, or 64 + the first
      // interchange that names the same outside row
      const int p = s_piv[tid];
      int first = tid;
#pragma unroll 16
      for (int k = kInvNB - 1; k >= 0; --k)
        if (k < tid && s_piv[k] == p) first = k;
      const bool inside = p < j0 + kInvNB;
      s_slot[tid] = inside ? p - j0 : kInvNB + first;
      s_row[tid] = (tid < nb) ? j0 + tid : -1;
      s_row[kInvNB + tid] = (!inside && first == tid) ? p : -1;
    }
  } else if (tid < kInvNB) {
    s_row[tid] = (tid < nb) ? j0 + tid : -1;
  }
  if (solve) {
#pragma unroll
    for (int u = 0; u < kBrLoads; ++u) {
      const int e = tid + u * kBrThreads;
      const int i = e / kInvNB, k = e % kInvNB;
      t[u] = (i < nb && k < nb) ? __ldcg(g.lu + (int64_t)(j0 + i) * n + j0 + k)
                                : (i == k ? 1.0f : 0.0f);
    }
  }
  __syncthreads();
  // all loads of a batch are issued before the first value is stored
#pragma unroll
  for (int h = 0; h < kRows / kInvNB; ++h) {
    float v[kBrLoads];
#pragma unroll
    for (int u = 0; u < kBrLoads; ++u) {
      const int e = tid + u * kBrThreads, i = h * kInvNB + e / kBrCols, c = e % kBrCols;
      const int row = s_row[i];
      v[u] = (row >= 0 && c0 + c < cend) ? __ldcg(g.w + (int64_t)row * n + c0 + c) : 0.0f;
    }
#pragma unroll
    for (int u = 0; u < kBrLoads; ++u) {
      const int e = tid + u * kBrThreads;
      X[h * kInvNB + e / kBrCols][e % kBrCols] = v[u];
    }
  }
  if (solve) {
#pragma unroll
    for (int u = 0; u < kBrLoads; ++u) {
      const int e = tid + u * kBrThreads;
      Tt[e % kInvNB][e / kInvNB] = t[u];
    }
  }
  __syncthreads();
  if (KIND == 0) {
    if (tid < kBrCols) {
#pragma unroll 8
      for (int k = 0; k < nb; ++k) {
        const int sl = s_slot[k];
        const float u = X[k][tid], v = X[sl][tid];
        X[k][tid] = v;
        X[sl][tid] = u;
      }
    }
    __syncthreads();
  }
  if (solve && tid < kBrCols) {
    // Each thread substitutes its own column, 16 rows at a time in registers:
    // one body for the product with a 16 x 16 block and one for the triangle.
#pragma unroll 1
    for (int bi = 0; bi < kInvNB / kBrT; ++bi) {
      const int i0 = (KIND != 2) ? bi * kBrT : kInvNB - kBrT - bi * kBrT;
      float x[kBrT];
#pragma unroll
      for (int i = 0; i < kBrT; ++i) x[i] = X[i0 + i][tid];
#pragma unroll 1
      for (int bk = 0; bk < bi; ++bk) {
        const int k0 = (KIND != 2) ? bk * kBrT : kInvNB - kBrT - bk * kBrT;
        float xk[kBrT];
#pragma unroll
        for (int k = 0; k < kBrT; ++k) xk[k] = X[k0 + k][tid];
#pragma unroll
        for (int kk = 0; kk < kBrT; ++kk) {
          const int k = (KIND != 2) ? kk : kBrT - 1 - kk;
#pragma unroll
          for (int i4 = 0; i4 < kBrT / 4; ++i4) {
            const float4 tq = *reinterpret_cast<const float4*>(&Tt[k0 + k][i0 + 4 * i4]);
            x[4 * i4 + 0] = fmaf(-tq.x, xk[k], x[4 * i4 + 0]);
            x[4 * i4 + 1] = fmaf(-tq.y, xk[k], x[4 * i4 + 1]);
            x[4 * i4 + 2] = fmaf(-tq.z, xk[k], x[4 * i4 + 2]);
            x[4 * i4 + 3] = fmaf(-tq.w, xk[k], x[4 * i4 + 3]);
          }
        }
      }
#pragma unroll
      for (int kk = 0; kk < kBrT; ++kk) {
        const int k = (KIND != 2) ? kk : kBrT - 1 - kk;
        if (KIND == 2) x[k] = x[k] / Tt[i0 + k][i0 + k];
        const float xk = x[k];
#pragma unroll
        for (int i4 = 0; i4 < kBrT / 4; ++i4) {
          if ((KIND != 2) ? (4 * i4 + 3 <= k) : (4 * i4 >= k)) continue;
          const float4 tq = *reinterpret_cast<const float4*>(&Tt[i0 + k][i0 + 4 * i4]);
          const float t4[4] = {tq.x, tq.y, tq.z, tq.w};
#pragma unroll
          for (int q = 0; q < 4; ++q)
            if ((KIND != 2) ? (4 * i4 + q > k) : (4 * i4 + q < k))
              x[4 * i4 + q] = fmaf(-t4[q], xk, x[4 * i4 + q]);
        }
      }
#pragma unroll
      for (int i = 0; i < kBrT; ++i) X[i0 + i][tid] = x[i];
    }
  }
  __syncthreads();
#pragma unroll 16
  for (int u = 0; u < kRows * kBrCols / kBrThreads; ++u) {
    const int e = tid + u * kBrThreads, i = e / kBrCols, c = e % kBrCols;
    const int row = s_row[i];
    if (row >= 0 && c0 + c < cend) g.w[(int64_t)row * n + c0 + c] = X[i][c];
  }
  if (solve) {
    // transposed copy, coalesced along the 64 entries of each column
#pragma unroll 16
    for (int u = 0; u < kInvNB * kBrCols / kBrThreads; ++u) {
      const int e = tid + u * kBrThreads, c = e / kInvNB, i = e % kInvNB;
      if (c0 + c < cend)
        br_store<PREC>(g.b0, g.b1, (int64_t)(c0 + c - g.c_begin) * kInvNB + i, X[i][c]);
    }
  }
}

template <int KIND>
static int launch_block_row(int prec, BlockRowArgs g, cudaStream_t st) {
  const int cols = g.c_end - g.c_begin;
  g.left = KIND == 0 ? (g.j0 + kBrCols - 1) / kBrCols : 0;
  g.strips = g.left + (cols + kBrCols - 1) / kBrCols;
  const int others = prec != 0 ? (g.na + kInvNB - 1) / kInvNB : 0;
  if (g.strips + others == 0) return LXGB_SUCCESSFUL;
  // (the inversions have no BF16 form)
  auto fn = prec == 0 ? block_row_kernel<KIND, 0>
                      : (KIND != 0 || prec == 1 ? block_row_kernel<KIND, 1>
                                                : block_row_kernel<KIND, KIND == 0 ? 2 : 1>);
  const int rows = KIND == 0 ? 2 * kInvNB : kInvNB;
  const int smem = (kInvNB * (kInvNB + 4) + rows * kBrLd) * (int)sizeof(float);
  LXGB_CUDA_TRY(ensure_dynamic_smem(reinterpret_cast<const void*>(fn), smem), "block_row: set smem");
  LXGB_CUDA_TRY(launch_pdl(fn, dim3((unsigned)(g.strips + others)), dim3(kBrThreads), (size_t)smem,
                           st, 1, g),
                "block_row: launch");
  return check_launch("block_row");
}

// ---------------------------------------------------------------------------
// FP32 products (x rounded to FP32).  TRI 0 full; 1 lower (columns < the row
// block's end: the matrix holds zeros above its diagonal); 2 upper (columns from
// the row block's start).  OUT 0: yh; 1: y64 = value; 2: y64 = b64 - value.
// A CTA owns 16 rows and 16 right-hand sides; its eight warps each keep 4 rows x
// 8 right-hand sides of accumulators while the lanes walk the columns, then
// reduce across lanes.
// ---------------------------------------------------------------------------
template <int TRI, int OUT>
__global__ void __launch_bounds__(256, 2)
gemv16_kernel(int m, int ncol, const float* __restrict__ Mh, int64_t ldm, int k,
              const float* __restrict__ xh, int64_t ldx, float* __restrict__ yh,
              double* __restrict__ y64, const double* __restrict__ b64, int64_t ldy) {
  const int nblk = (m + kGvRows - 1) / kGvRows;
  // Lower triangles: the heaviest row blocks (last) start first.
  const int rb = (TRI == 1) ? (nblk - 1 - (int)blockIdx.x) : (int)blockIdx.x;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int row0 = rb * kGvRows + (warp & 3) * 4;
  const int rhs0 = (int)blockIdx.y * kGvRhs + (warp >> 2) * 8;
  int c_lo = 0, c_hi = ncol;
  if (TRI == 1) c_hi = min(ncol, rb * kGvRows + kGvRows);
  if (TRI == 2) c_lo = rb * kGvRows;

  // Rows and right-hand sides past the ends are clamped to the last valid
  // one (in-bounds loads; their results are never written).
  const float* mr[4];
#pragma unroll
  for (int r = 0; r < 4; ++r) mr[r] = Mh + (int64_t)min(row0 + r, m - 1) * ldm;
  int xo[8];
#pragma unroll
  for (int q = 0; q < 8; ++q) xo[q] = min(rhs0 + q, k - 1) * (int)ldx;
  float ah[4][8];
#pragma unroll
  for (int r = 0; r < 4; ++r)
#pragma unroll
    for (int q = 0; q < 8; ++q) ah[r][q] = 0.0f;
  for (int c = c_lo + lane; c < c_hi; c += 32) {
    float mv[4], xv[8];
#pragma unroll
    for (int r = 0; r < 4; ++r) mv[r] = __ldg(mr[r] + c);
#pragma unroll
    for (int q = 0; q < 8; ++q) xv[q] = __ldg(xh + c + xo[q]);
#pragma unroll
    for (int q = 0; q < 8; ++q)
#pragma unroll
      for (int r = 0; r < 4; ++r) ah[r][q] = fmaf(mv[r], xv[q], ah[r][q]);
  }
  // Butterfly reduction across the lanes (every lane ends with every sum).
#pragma unroll
  for (int off = 16; off > 0; off >>= 1)
#pragma unroll
    for (int r = 0; r < 4; ++r)
#pragma unroll
      for (int q = 0; q < 8; ++q) ah[r][q] += __shfl_xor_sync(0xffffffffu, ah[r][q], off);
  // Lane r*8 + q writes (row0 + r, rhs0 + q).
  float oh = 0.0f;
#pragma unroll
  for (int r = 0; r < 4; ++r)
#pragma unroll
    for (int q = 0; q < 8; ++q)
      if (lane == r * 8 + q) oh = ah[r][q];
  const int row = row0 + (lane >> 3), rhs = rhs0 + (lane & 7);
  if (row >= m || rhs >= k) return;
  const int64_t o = (int64_t)rhs * ldy + row;
  if (OUT == 0) {
    yh[o] = oh;
  } else {
    const double v = (double)oh;
    y64[o] = (OUT == 2) ? b64[o] - v : v;
  }
}

// ---------------------------------------------------------------------------
// Double-float products Y = T X, T exact FP32 or a hi + lo pair (LO), X a pair:
// a CTA owns 32 rows x NR right-hand sides, a cluster of CTAs splits the columns.
//
// What bounds it is the FP32 pipe.  A multiply-add takes 10 operations (9
// without lo): p = fl(a x), r = fl(s + p), and as in TwoSum z = r - s,
// t = r - z, whose exact parts give s + p - r = (s - t) + (p - z); the
// product's own rounding error joins the second part, (p - z) + (a x - p) =
// a x - z, in one FMA.  (TwoProd and TwoSum apart take 12.)  The FMA's rounding
// is 2^-24 of a term that is itself at most an ulp; measured against 128 bits,
// the sums' errors are those of the 12-operation form.  The low-order terms
// join by FMAs before the one addition to the second accumulator.
// A thread keeps 4 rows x NR/4 right-hand sides; the operands are staged by
// asynchronous copies, 64 columns at a time, and the eight warps take the
// columns of a stage in pairs (8-byte loads from shared memory).  The warps' and
// then the cluster's partial sums are added in a fixed order.
// Measured, n = 8192, 16 right-hand sides: hi + lo matrix 396 us (one CTA of 16
// rows per SM, loads and sums one column at a time: 877 us), triangles 186 us
// (329): 57 % of the FP32 pipe's rate.
// ---------------------------------------------------------------------------
constexpr int kDfRows = 32;     // rows per CTA
constexpr int kDfK = 64;        // columns per stage
constexpr int kDfLd = kDfK + 4; // padded row: 16-byte aligned, conflict-free over 8 rows
constexpr int kDfThreads = 256;

// `bytes` of the 4 VEC bytes at src (the rest zero) into shared memory.
template <int VEC>
__device__ __forceinline__ void df_copy(float* dst, const float* src, int bytes) {
  const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
  if (VEC == 4)
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(src), "r"(bytes)
                 : "memory");
  else
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(d), "l"(src), "r"(bytes)
                 : "memory");
}

template <int NR, bool LO>
constexpr size_t df_stage_floats() {
  return (size_t)((LO ? 2 : 1) * kDfRows + 2 * NR) * kDfLd;
}
template <int NR, bool LO>
constexpr size_t df_smem() {
  return 2 * df_stage_floats<NR, LO>() * sizeof(float);
}

template <int NR, bool LO, int TRI, int OUT, int VEC>
__global__ void __launch_bounds__(kDfThreads, 2)
gemm_df_kernel(int m, int ncol, const float* __restrict__ Mh, const float* __restrict__ Ml,
               int64_t ldm, int k, const float* __restrict__ xh, const float* __restrict__ xl,
               int64_t ldx, float* __restrict__ yh, float* __restrict__ yl,
               double* __restrict__ y64, const double* __restrict__ b64, int64_t ldy) {
  constexpr int J = NR / 4;                 // right-hand sides per thread
  constexpr int kOut = kDfRows * NR;
  extern __shared__ __align__(16) float df_dyn[];
  __shared__ float2 pub[kOut];
  cg::cluster_group cluster = cg::this_cluster();
  const int parts = (int)cluster.num_blocks();
  const int part = (int)cluster.block_rank();
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int rg = lane & 7, cgp = lane >> 3;
  const int nblk = (m + kDfRows - 1) / kDfRows;
  const int bx = (int)(blockIdx.x / parts);
  // lower triangles: the heaviest row blocks (last) start first
  const int rb = (TRI == 1) ? (nblk - 1 - bx) : bx;
  const int row0 = rb * kDfRows;
  const int rhs0 = (int)blockIdx.y * NR;
  int c_lo = 0, c_hi = ncol;
  if (TRI == 1) c_hi = min(ncol, row0 + kDfRows);
  if (TRI == 2) c_lo = row0;                // a multiple of 32: stages start aligned
  const int chunks = (c_hi - c_lo + kDfK - 1) / kDfK;
  const int ch0 = (int)((int64_t)chunks * part / parts);
  const int ch1 = (int)((int64_t)chunks * (part + 1) / parts);
  auto stage = [&](int buf) { return df_dyn + buf * df_stage_floats<NR, LO>(); };
  auto load = [&](int ch, int buf) {
    float* A = stage(buf);
    float* X = A + (LO ? 2 : 1) * kDfRows * kDfLd;
    constexpr int kPer = kDfK / VEC;        // copies per row
    const int cb = c_lo + ch * kDfK;
#pragma unroll
    for (int e0 = 0; e0 < kDfRows * kPer; e0 += kDfThreads) {
      const int e = e0 + tid;
      const int r = e / kPer, c = (e % kPer) * VEC;
      const int left = (row0 + r < m) ? min(VEC, max(0, c_hi - cb - c)) * 4 : 0;
      const int64_t o = left ? (int64_t)(row0 + r) * ldm + cb + c : 0;
      df_copy<VEC>(A + r * kDfLd + c, Mh + o, left);
      if (LO) df_copy<VEC>(A + (kDfRows + r) * kDfLd + c, Ml + o, left);
    }
    for (int e = tid; e < NR * kPer; e += kDfThreads) {
      const int r = e / kPer, c = (e % kPer) * VEC;
      const int left = (rhs0 + r < k) ? min(VEC, max(0, c_hi - cb - c)) * 4 : 0;
      const int64_t o = left ? (int64_t)(rhs0 + r) * ldx + cb + c : 0;
      df_copy<VEC>(X + r * kDfLd + c, xh + o, left);
      df_copy<VEC>(X + (NR + r) * kDfLd + c, xl + o, left);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  float s[4][J], sl[4][J];
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < J; ++j) s[i][j] = sl[i][j] = 0.0f;
  if (ch0 < ch1) load(ch0, 0);
  for (int ch = ch0; ch < ch1; ++ch) {
    const int buf = (ch - ch0) & 1;
    if (ch + 1 < ch1) {
      load(ch + 1, buf ^ 1);
      asm volatile("cp.async.wait_group 1;" ::: "memory");
    } else {
      asm volatile("cp.async.wait_group 0;" ::: "memory");
    }
    __syncthreads();
    const float* A = stage(buf);
    const float* X = A + (LO ? 2 : 1) * kDfRows * kDfLd;
#pragma unroll
    for (int u = 0; u < kDfK / 16; ++u) {
      const int c = 2 * (warp + 8 * u);
      float2 a[4], al[4], x[J], x2[J];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        a[i] = *reinterpret_cast<const float2*>(A + (8 * i + rg) * kDfLd + c);
        al[i] = LO ? *reinterpret_cast<const float2*>(A + (kDfRows + 8 * i + rg) * kDfLd + c)
                   : make_float2(0.f, 0.f);
      }
#pragma unroll
      for (int j = 0; j < J; ++j) {
        x[j] = *reinterpret_cast<const float2*>(X + (4 * j + cgp) * kDfLd + c);
        x2[j] = *reinterpret_cast<const float2*>(X + (NR + 4 * j + cgp) * kDfLd + c);
      }
#pragma unroll
      for (int j = 0; j < J; ++j)
#pragma unroll
        for (int i = 0; i < 4; ++i) df_mac<LO>(s[i][j], sl[i][j], a[i].x, al[i].x, x[j].x, x2[j].x);
#pragma unroll
      for (int j = 0; j < J; ++j)
#pragma unroll
        for (int i = 0; i < 4; ++i) df_mac<LO>(s[i][j], sl[i][j], a[i].y, al[i].y, x[j].y, x2[j].y);
    }
    __syncthreads();
  }
  // warps: output o = rhs * 32 + row (the staging buffers are free now)
  float2* red = reinterpret_cast<float2*>(df_dyn);  // [8][kOut]
  static_assert(8 * kOut * sizeof(float2) <= df_smem<NR, LO>(), "reduction fits the stages");
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < J; ++j)
      red[warp * kOut + (4 * j + cgp) * kDfRows + 8 * i + rg] = make_float2(s[i][j], sl[i][j]);
  __syncthreads();
  for (int o = tid; o < kOut; o += kDfThreads) {
    float2 v = red[o];
#pragma unroll
    for (int w = 1; w < 8; ++w) {
      const float2 u = red[w * kOut + o];
      float err;
      two_sum(v.x, u.x, err);
      v.y += u.y + err;
    }
    pub[o] = v;
  }
  cluster.sync();
  // the cluster: CTA `part` finishes its share of the outputs
  const int share = kOut / parts;
  for (int q = tid; q < share; q += kDfThreads) {
    const int o = part * share + q;
    float2 v = cluster.map_shared_rank(pub, 0)[o];
    for (int c = 1; c < parts; ++c) {
      const float2 u = cluster.map_shared_rank(pub, c)[o];
      float err;
      two_sum(v.x, u.x, err);
      v.y += u.y + err;
    }
    const int row = row0 + o % kDfRows, rhs = rhs0 + o / kDfRows;
    if (row < m && rhs < k) {
      float e;
      fast_two_sum(v.x, v.y, e);
      const int64_t at = (int64_t)rhs * ldy + row;
      if (OUT == 0) {
        yh[at] = v.x;
        yl[at] = e;
      } else {
        const double d = (double)v.x + (double)e;
        y64[at] = (OUT == 2) ? b64[at] - d : d;
      }
    }
  }
  cluster.sync();  // no CTA leaves while another may still read its sums
}

template <int NR, bool LO, int TRI, int OUT, int VEC>
static int launch_df_nr(int m, int ncol, const float* Mh, const float* Ml, int64_t ldm, int k,
                        const float* xh, const float* xl, int64_t ldx, float* yh, float* yl,
                        double* y64, const double* b64, int64_t ldy, cudaStream_t st) {
  auto fn = gemm_df_kernel<NR, LO, TRI, OUT, VEC>;
  const int nblk = (m + kDfRows - 1) / kDfRows;
  // columns split so that about 1000 CTAs share the SMs evenly (256 row blocks
  // alone would leave 48 SMs with two and 104 with one at a time)
  const int parts = nblk <= 128 ? 8 : (nblk <= 256 ? 4 : 2);
  constexpr size_t smem = df_smem<NR, LO>();
  LXGB_CUDA_TRY(ensure_dynamic_smem(reinterpret_cast<const void*>(fn), (int)smem), "gemm_df: smem");
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(nblk * parts), (unsigned)((k + NR - 1) / NR));
  cfg.blockDim = dim3(kDfThreads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = (unsigned)parts;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  LXGB_CUDA_TRY(cudaLaunchKernelEx(&cfg, fn, m, ncol, Mh, Ml, ldm, k, xh, xl, ldx, yh, yl, y64,
                                   b64, ldy),
                "gemm_df: launch");
  return check_launch("gemm_df");
}

// 4, 8 or 16 right-hand sides per CTA; 16-byte copies when every row of the
// operands starts on a 16-byte boundary.
template <bool LO, int TRI, int OUT>
static int launch_df(int m, int ncol, const float* Mh, const float* Ml, int64_t ldm, int k,
                     const float* xh, const float* xl, int64_t ldx, float* yh, float* yl,
                     double* y64, const double* b64, int64_t ldy, cudaStream_t st) {
  if (m <= 0 || k <= 0) return LXGB_SUCCESSFUL;
  const bool vec = (((uintptr_t)Mh | (uintptr_t)(LO ? Ml : Mh) | (uintptr_t)xh | (uintptr_t)xl) &
                    15) == 0 &&
                   (ldm & 3) == 0 && (ldx & 3) == 0;
#define LXGB_DF(NR)                                                                              \
  return vec ? launch_df_nr<NR, LO, TRI, OUT, 4>(m, ncol, Mh, Ml, ldm, k, xh, xl, ldx, yh, yl,   \
                                                 y64, b64, ldy, st)                              \
             : launch_df_nr<NR, LO, TRI, OUT, 1>(m, ncol, Mh, Ml, ldm, k, xh, xl, ldx, yh, yl,   \
                                                 y64, b64, ldy, st)
  if (k <= 4) LXGB_DF(4);
  if (k <= 8) LXGB_DF(8);
  LXGB_DF(16);
#undef LXGB_DF
}

// Few right-hand sides (k <= 4): one warp per matrix row, lanes along the
// columns, k double-float accumulators per lane reduced across the warp.
// The matrix streams from HBM once; x (hi/lo, k × n) is shared through L1/L2.
template <int K, bool LO, int OUT>
__global__ void __launch_bounds__(256)
gemv_rows_df_kernel(int m, int ncol, const float* __restrict__ Mh, const float* __restrict__ Ml,
                    int64_t ldm, const float* __restrict__ xh, const float* __restrict__ xl,
                    int64_t ldx, double* __restrict__ y64, const double* __restrict__ b64,
                    int64_t ldy) {
  const int lane = threadIdx.x & 31;
  const int row = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (row >= m) return;  // whole warps
  const float* mr = Mh + (int64_t)row * ldm;
  const float* ml = LO ? Ml + (int64_t)row * ldm : mr;
  float sh[K], sl[K];
#pragma unroll
  for (int q = 0; q < K; ++q) sh[q] = sl[q] = 0.0f;
  auto step = [&](float a, float al, int q, float x, float xlv) {
    const float p = a * x;
    float e = fmaf(a, x, -p);
    e = fmaf(a, xlv, e);
    if (LO) e = fmaf(al, x, e);
    float err;
    two_sum(sh[q], p, err);
    sl[q] += err + e;
  };
  // 16-byte loads, two groups of 128 columns in flight, where every row of the
  // matrix and of x starts on a 16-byte boundary (one column per lane and
  // iteration ran at a sixth of the HBM rate: 238 us for 2048 x 16384)
  int c = 0;
  if ((((uintptr_t)Mh | (uintptr_t)(LO ? Ml : Mh) | (uintptr_t)xh | (uintptr_t)xl) & 15) == 0 &&
      (ldm & 3) == 0 && (ldx & 3) == 0) {
#pragma unroll 2
    for (; c + 128 <= ncol; c += 128) {
      const int o = c + 4 * lane;
      const float4 a = __ldg(reinterpret_cast<const float4*>(mr + o));
      const float4 al = LO ? __ldg(reinterpret_cast<const float4*>(ml + o))
                           : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
      for (int q = 0; q < K; ++q) {
        const float4 x = __ldg(reinterpret_cast<const float4*>(xh + (int64_t)q * ldx + o));
        const float4 xlv = __ldg(reinterpret_cast<const float4*>(xl + (int64_t)q * ldx + o));
        step(a.x, al.x, q, x.x, xlv.x);
        step(a.y, al.y, q, x.y, xlv.y);
        step(a.z, al.z, q, x.z, xlv.z);
        step(a.w, al.w, q, x.w, xlv.w);
      }
    }
  }
  for (c += lane; c < ncol; c += 32) {
    const float a = __ldg(mr + c);
    const float al = LO ? __ldg(ml + c) : 0.0f;
#pragma unroll
    for (int q = 0; q < K; ++q)
      step(a, al, q, __ldg(xh + (int64_t)q * ldx + c), __ldg(xl + (int64_t)q * ldx + c));
  }
#pragma unroll
  for (int off = 16; off > 0; off >>= 1)
#pragma unroll
    for (int q = 0; q < K; ++q) {
      const float oh = __shfl_xor_sync(0xffffffffu, sh[q], off);
      const float ol = __shfl_xor_sync(0xffffffffu, sl[q], off);
      float err;
      two_sum(sh[q], oh, err);
      sl[q] += ol + err;
    }
  if (lane < K) {
    float oh = sh[0], ol = sl[0];
#pragma unroll
    for (int q = 1; q < K; ++q)
      if (lane == q) { oh = sh[q]; ol = sl[q]; }
    const double v = (double)oh + (double)ol;
    const int64_t o = (int64_t)lane * ldy + row;
    y64[o] = (OUT == 2) ? b64[o] - v : v;
  }
}

template <int K, bool LO>
static void launch_rows_df(int m, int n, const float* ah, const float* al, int64_t lda,
                           const float* xh, const float* xl, int64_t ldx, double* y,
                           const double* b, int64_t ldy, cudaStream_t st) {
  const unsigned g = (unsigned)((m + 7) / 8);
  if (b)
    gemv_rows_df_kernel<K, LO, 2><<<g, 256, 0, st>>>(m, n, ah, al, lda, xh, xl, ldx, y, b, ldy);
  else
    gemv_rows_df_kernel<K, LO, 1><<<g, 256, 0, st>>>(m, n, ah, al, lda, xh, xl, ldx, y, b, ldy);
}

// zh/zl[q][i] = x[q][perm ? perm[i] : i] as a hi + lo pair (zl null: FP32 rounding).
__global__ void split_rows_kernel(int k, int n, const double* __restrict__ x, int64_t ldx,
                                  const int32_t* __restrict__ perm, float* __restrict__ zh,
                                  float* __restrict__ zl, int64_t ldz) {
  const int64_t total = (int64_t)k * n;
  for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < total;
       e += (int64_t)gridDim.x * blockDim.x) {
    const int q = (int)(e / n), i = (int)(e % n);
    const double v = x[(int64_t)q * ldx + (perm ? perm[i] : i)];
    if (zl) {
      float h, l;
      split_f64(v, h, l);
      zh[(int64_t)q * ldz + i] = h;
      zl[(int64_t)q * ldz + i] = l;
    } else {
      zh[(int64_t)q * ldz + i] = __double2float_rn(v);
    }
  }
}

// One CTA per row at a time, two columns per thread and step (16-byte loads)
// where the rows start on 16-byte boundaries, values taken as 32-bit words: as
// doubles, the loads' zero fills and the rare conversions' selects ran on the
// FP64 pipe for every element (380 us for 16384 x 2048).
template <bool VEC>
__global__ void __launch_bounds__(256)
split_matrix_kernel(int64_t rows, int64_t cols, const double* __restrict__ a, int64_t lda,
                    float* __restrict__ hi, float* __restrict__ lo, int64_t ld) {
  for (int64_t r = blockIdx.x; r < rows; r += gridDim.x) {
    const uint2* ar = reinterpret_cast<const uint2*>(a + r * lda);
    float* hr = hi + r * ld;
    float* lr = lo ? lo + r * ld : nullptr;
    const int64_t even = VEC ? (cols & ~(int64_t)1) : 0;  // columns taken in pairs
#pragma unroll 4
    for (int64_t c = 2 * threadIdx.x; c < even; c += 512) {
      const uint4 v = *reinterpret_cast<const uint4*>(ar + c);
      const uint2 w[2] = {make_uint2(v.x, v.y), make_uint2(v.z, v.w)};
      float h[2], l[2];
      splitw<2>(w, h, l);
      *reinterpret_cast<float2*>(hr + c) = make_float2(h[0], h[1]);
      if (lr) *reinterpret_cast<float2*>(lr + c) = make_float2(l[0], l[1]);
    }
    for (int64_t c = even + threadIdx.x; c < cols; c += 256) {
      const uint2 w[1] = {ar[c]};
      float h[1], l[1];
      splitw<1>(w, h, l);
      hr[c] = h[0];
      if (lr) lr[c] = l[0];
    }
  }
}

template <int TRI, int OUT>
int launch_gemv16(int m, int ncol, const float* Mh, int64_t ldm, int k, const float* xh,
                  int64_t ldx, float* yh, double* y64, const double* b64, int64_t ldy,
                  cudaStream_t st) {
  LXGB_REQUIRE((int64_t)k * ldx < ((int64_t)1 << 31), "gemv16: right-hand-side block above 2^31 entries");
  dim3 grid((unsigned)((m + kGvRows - 1) / kGvRows), (unsigned)((k + kGvRhs - 1) / kGvRhs));
  gemv16_kernel<TRI, OUT><<<grid, 256, 0, st>>>(m, ncol, Mh, ldm, k, xh, ldx, yh, y64, b64, ldy);
  return check_launch("gemv16");
}

int lu32_block_row(int precision, int n, int j0, int nb, float* lu, const int32_t* piv, void* a0,
                   void* a1, void* b0, void* b1, cudaStream_t st) {
  BlockRowArgs g = {};
  g.n = n;
  g.j0 = j0;
  g.nb = nb;
  g.lu = lu;
  g.w = lu;
  g.piv = piv;
  g.c_begin = j0 + nb;
  g.c_end = n;
  g.b0 = b0;
  g.b1 = b1;
  g.a_src = lu + (int64_t)(j0 + nb) * n + j0;
  g.na = n - j0 - nb;
  g.a0 = a0;
  g.a1 = a1;
  return launch_block_row<0>(precision, g, st);
}

static int64_t blk_bytes(int n) {
  return (((int64_t)(n > 0 ? n : 1) * kInvNB * (int64_t)sizeof(float)) + 255) & ~(int64_t)255;
}

static int64_t vec_bytes(int n, int nrhs) {
  return (((int64_t)(n > 0 ? n : 1) * (nrhs > 0 ? nrhs : 1) * (int64_t)sizeof(float)) + 255) &
         ~(int64_t)255;
}

}  // namespace lxgb

using namespace lxgb;

extern "C" int64_t lxgb_lu32_inverse_workspace_size(int32_t n, int32_t precision) {
  // the update's operands, one set for each of the two inverses
  return 256 + 2 * (precision == 1 ? 5 : 1) * blk_bytes(n);
}

extern "C" int lxgb_lu32_inverse(int32_t n, const float* lu, const int32_t* piv, float* linv,
                                 float* uinv, int32_t* perm, int32_t precision, int32_t* err,
                                 void* work, int64_t work_bytes, void* stream) {
  LXGB_REQUIRE(precision == 0 || precision == 1, "lu32_inverse: precision must be 0 or 1");
  LXGB_REQUIRE(n >= 0, "lu32_inverse: negative size");
  if (n == 0) return LXGB_SUCCESSFUL;
  LXGB_REQUIRE(n <= kPermMaxN, "lu32_inverse: n above 25600");
  LXGB_REQUIRE(lu && piv && (linv || uinv) && perm && err && work,
               "lu32_inverse: null pointer");
  LXGB_REQUIRE((n % 4) == 0, "lu32_inverse: n must be a multiple of 4 (16-byte TMA rows)");
  LXGB_REQUIRE((((uintptr_t)lu) & 15) == 0 && (((uintptr_t)work) & 255) == 0,
               "lu32_inverse: lu must be 16-byte and work 256-byte aligned");
  if (work_bytes < lxgb_lu32_inverse_workspace_size(n, precision)) {
    set_last_error("lu32_inverse: workspace too small");
    return LXGB_WORKSPACE_TOO_SMALL;
  }
  cudaStream_t st = as_stream(stream);
  const size_t psmem = (size_t)2 * n * sizeof(int32_t);
  LXGB_CUDA_TRY(ensure_dynamic_smem(reinterpret_cast<const void*>(perm_from_swaps_kernel), (int)psmem),
                "lu32_inverse: set smem");
  perm_from_swaps_kernel<<<1, 1024, psmem, st>>>(n, piv, perm);
  const unsigned idg = (unsigned)(n < 4096 ? n : 4096);
  if (linv) set_identity_f32_kernel<<<idg, 256, 0, st>>>(n, linv);
  if (uinv) set_identity_f32_kernel<<<idg, 256, 0, st>>>(n, uinv);
  const int64_t blk = blk_bytes(n);
  const bool split = precision == 1;
  // operands of an inverse's update: a hi, lo; X^T hi (or FP32), lo
  struct Operands { float *ah, *al, *b, *bl; };
  auto operands = [&](int set) {
    char* p = reinterpret_cast<char*>(work) + 256 + (int64_t)set * (split ? 5 : 1) * blk;
    auto at = [&](int i) { return reinterpret_cast<float*>(p + i * blk); };
    return split ? Operands{at(1), at(2), at(3), at(4)} : Operands{nullptr, nullptr, at(0), nullptr};
  };
  const Operands ol = operands(0), ou = operands(1);
  auto block = [&](const Operands& o, float* w, int j0, int nb, int c_begin, int c_end,
                   const float* a_src, int na) {
    BlockRowArgs g = {};
    g.n = n;
    g.j0 = j0;
    g.nb = nb;
    g.lu = lu;
    g.w = w;
    g.c_begin = c_begin;
    g.c_end = c_end;
    g.b0 = o.b;
    g.b1 = o.bl;
    g.a_src = a_src;
    g.na = na;
    g.a0 = o.ah;
    g.a1 = o.al;
    return g;
  };
  auto update = [&](const Operands& o, int rows, int cols, int nb, const float* a_src, float* c,
                    int beside) {
    if (rows <= 0) return (int)LXGB_SUCCESSFUL;
    if (split)
      return gemm_tf32_nt_split(rows, cols, nb, o.ah, o.al, kInvNB, o.b, o.bl, kInvNB, c, n, -1.0f,
                                1.0f, err, st, beside);
    return gemm_tf32_nt(rows, cols, nb, a_src, n, o.b, kInvNB, c, n, -1.0f, 1.0f, err, st, beside);
  };
  // L^{-1} top to bottom: row block j of W = L^{-1} has nonzeros in columns
  // < j0 + nb only.  U^{-1} bottom to top: row block j has nonzeros in columns
  // >= j0 only.  Either may be NULL: the square QR needs only R^{-1}, and a
  // Cholesky factor forms U^{-1} from L^{-1} with lxgb_chol32_uinv.  Both together
  // go step by step, the update of one beside the other's block row: 0.88 ms at n =
  // 2048, 2.43 at 4096, 9.2 at 8192, against 1.40, 3.27 and 10.5 one after the other.
  const int steps = (n + kInvNB - 1) / kInvNB;
  auto update_l = [&](int s, int beside) {
    const int j0 = s * kInvNB, nb = min(kInvNB, n - j0), ncols = j0 + nb;
    return update(ol, n - ncols, ncols, nb, lu + (int64_t)ncols * n + j0,
                  linv + (int64_t)ncols * n, beside);
  };
  auto update_u = [&](int s, int beside) {
    const int j0 = (steps - 1 - s) * kInvNB, nb = min(kInvNB, n - j0);
    return update(ou, j0, n - j0, nb, lu + j0, uinv + j0, beside);
  };
  for (int s = 0; s < steps; ++s) {
    int rc = LXGB_SUCCESSFUL;
    if (linv) {
      const int j0 = s * kInvNB, nb = min(kInvNB, n - j0), ncols = j0 + nb;
      rc = launch_block_row<1>(precision, block(ol, linv, j0, nb, 0, ncols,
                                                lu + (int64_t)ncols * n + j0, n - ncols), st);
      if (!rc && uinv && s > 0) rc = update_u(s - 1, kBesideRow);
      if (!rc && !uinv) rc = update_l(s, 0);
    }
    if (!rc && uinv) {
      const int j0 = (steps - 1 - s) * kInvNB, nb = min(kInvNB, n - j0);
      rc = launch_block_row<2>(precision, block(ou, uinv, j0, nb, j0, n, lu + j0, j0), st);
      if (!rc) rc = linv ? update_l(s, kBesideRow) : update_u(s, 0);
    }
    if (rc) return rc;
  }
  return check_launch("lu32_inverse");
}

extern "C" int64_t lxgb_lu32_apply_workspace_size(int32_t n, int32_t nrhs) {
  return 4 * vec_bytes(n, nrhs);
}

extern "C" int lxgb_lu32_apply(int32_t n, int32_t nrhs, const float* linv, const float* uinv,
                               const int32_t* perm, int32_t mode, const double* x, double* y,
                               void* work, int64_t work_bytes, void* stream) {
  LXGB_REQUIRE(mode == 0 || mode == 1, "lu32_apply: mode must be 0 (FP32) or 1 (double-float)");
  LXGB_REQUIRE(n >= 0 && nrhs >= 0, "lu32_apply: negative size");
  if (n == 0 || nrhs == 0) return LXGB_SUCCESSFUL;
  LXGB_REQUIRE(linv && uinv && perm && x && y && work, "lu32_apply: null pointer");
  if (work_bytes < lxgb_lu32_apply_workspace_size(n, nrhs)) {
    set_last_error("lu32_apply: workspace too small");
    return LXGB_WORKSPACE_TOO_SMALL;
  }
  cudaStream_t st = as_stream(stream);
  const int64_t vb = vec_bytes(n, nrhs);
  char* wb = reinterpret_cast<char*>(work);
  float* zh = reinterpret_cast<float*>(wb);
  float* zl = reinterpret_cast<float*>(wb + vb);
  float* th = reinterpret_cast<float*>(wb + 2 * vb);
  float* tl = reinterpret_cast<float*>(wb + 3 * vb);
  const int64_t total = (int64_t)n * nrhs;
  const unsigned g = (unsigned)((total + 255) / 256 < 4096 ? (total + 255) / 256 : 4096);
  split_rows_kernel<<<g, 256, 0, st>>>(nrhs, n, x, n, perm, zh, mode ? zl : nullptr, n);
  int rc;
  if (mode == 0) {
    rc = launch_gemv16<1, 0>(n, n, linv, n, nrhs, zh, n, th, nullptr, nullptr, n, st);
    if (!rc) rc = launch_gemv16<2, 1>(n, n, uinv, n, nrhs, th, n, nullptr, y, nullptr, n, st);
  } else {
    rc = launch_df<false, 1, 0>(n, n, linv, nullptr, n, nrhs, zh, zl, n, th, tl, nullptr, nullptr,
                                n, st);
    if (!rc)
      rc = launch_df<false, 2, 1>(n, n, uinv, nullptr, n, nrhs, th, tl, n, nullptr, nullptr, y,
                                  nullptr, n, st);
  }
  return rc;
}

extern "C" int64_t lxgb_qr32_apply_workspace_size(int32_t n, int32_t nrhs) {
  return 4 * vec_bytes(n, nrhs);
}

extern "C" int lxgb_qr32_apply(int32_t n, int32_t nrhs, const float* qt, const float* rinv,
                               int32_t mode, const double* x, double* y, void* work,
                               int64_t work_bytes, void* stream) {
  LXGB_REQUIRE(mode == 0 || mode == 1, "qr32_apply: mode must be 0 (FP32) or 1 (double-float)");
  LXGB_REQUIRE(n >= 0 && nrhs >= 0, "qr32_apply: negative size");
  if (n == 0 || nrhs == 0) return LXGB_SUCCESSFUL;
  LXGB_REQUIRE(qt && rinv && x && y && work, "qr32_apply: null pointer");
  if (work_bytes < lxgb_qr32_apply_workspace_size(n, nrhs)) {
    set_last_error("qr32_apply: workspace too small");
    return LXGB_WORKSPACE_TOO_SMALL;
  }
  cudaStream_t st = as_stream(stream);
  const int64_t vb = vec_bytes(n, nrhs);
  char* wb = reinterpret_cast<char*>(work);
  float* zh = reinterpret_cast<float*>(wb);
  float* zl = reinterpret_cast<float*>(wb + vb);
  float* th = reinterpret_cast<float*>(wb + 2 * vb);
  float* tl = reinterpret_cast<float*>(wb + 3 * vb);
  const int64_t total = (int64_t)n * nrhs;
  const unsigned g = (unsigned)((total + 255) / 256 < 4096 ? (total + 255) / 256 : 4096);
  split_rows_kernel<<<g, 256, 0, st>>>(nrhs, n, x, n, nullptr, zh, mode ? zl : nullptr, n);
  int rc;
  if (mode == 0) {
    rc = launch_gemv16<0, 0>(n, n, qt, n, nrhs, zh, n, th, nullptr, nullptr, n, st);
    if (!rc) rc = launch_gemv16<2, 1>(n, n, rinv, n, nrhs, th, n, nullptr, y, nullptr, n, st);
  } else {
    rc = launch_df<false, 0, 0>(n, n, qt, nullptr, n, nrhs, zh, zl, n, th, tl, nullptr, nullptr,
                                n, st);
    if (!rc)
      rc = launch_df<false, 2, 1>(n, n, rinv, nullptr, n, nrhs, th, tl, n, nullptr, nullptr, y,
                                  nullptr, n, st);
  }
  return rc;
}

extern "C" int lxgb_split_f64(int64_t rows, int64_t cols, const double* a, int64_t lda, float* hi,
                              float* lo, int64_t ld, void* stream) {
  LXGB_REQUIRE(rows >= 0 && cols >= 0, "split_f64: negative size");
  if (rows == 0 || cols == 0) return LXGB_SUCCESSFUL;
  LXGB_REQUIRE(a && hi, "split_f64: null pointer");
  LXGB_REQUIRE(lda >= cols && ld >= cols, "split_f64: leading dimension too small");
  const unsigned g = (unsigned)(rows < 65535 ? rows : 65535);
  const bool vec = (((uintptr_t)a) & 15) == 0 && (lda & 1) == 0 && (((uintptr_t)hi) & 7) == 0 &&
                   (((uintptr_t)lo) & 7) == 0 && (ld & 1) == 0;
  if (vec)
    split_matrix_kernel<true><<<g, 256, 0, as_stream(stream)>>>(rows, cols, a, lda, hi, lo, ld);
  else
    split_matrix_kernel<false><<<g, 256, 0, as_stream(stream)>>>(rows, cols, a, lda, hi, lo, ld);
  return check_launch("split_f64");
}

extern "C" int64_t lxgb_gemv_df_workspace_size(int32_t n, int32_t nrhs) {
  return 2 * vec_bytes(n, nrhs);
}

extern "C" int lxgb_gemv_df(int32_t m, int32_t n, const float* a_hi, const float* a_lo,
                            int64_t lda, int32_t nrhs, const double* x, int64_t ldx,
                            const double* b, double* y, int64_t ldy, int32_t mode, void* work,
                            int64_t work_bytes, void* stream) {
  LXGB_REQUIRE(mode == 0 || mode == 1, "gemv_df: mode must be 0 (FP32) or 1 (double-float)");
  LXGB_REQUIRE(m >= 0 && n >= 0 && nrhs >= 0, "gemv_df: negative size");
  if (m == 0 || nrhs == 0) return LXGB_SUCCESSFUL;
  LXGB_REQUIRE(a_hi && y && (n == 0 || x) && work, "gemv_df: null pointer");
  LXGB_REQUIRE(lda >= n && ldx >= n && ldy >= m, "gemv_df: leading dimension too small");
  if (work_bytes < lxgb_gemv_df_workspace_size(n, nrhs)) {
    set_last_error("gemv_df: workspace too small");
    return LXGB_WORKSPACE_TOO_SMALL;
  }
  cudaStream_t st = as_stream(stream);
  const int64_t vb = vec_bytes(n, nrhs);
  float* xh = reinterpret_cast<float*>(work);
  float* xl = reinterpret_cast<float*>(reinterpret_cast<char*>(work) + vb);
  const int nn = n > 0 ? n : 1;
  if (n > 0) {
    const int64_t total = (int64_t)n * nrhs;
    const unsigned g = (unsigned)((total + 255) / 256 < 4096 ? (total + 255) / 256 : 4096);
    split_rows_kernel<<<g, 256, 0, st>>>(nrhs, n, x, ldx, nullptr, xh, mode ? xl : nullptr, nn);
  }
  const bool res = b != nullptr;
  if (mode == 1 && nrhs <= 4 && n > 0) {
    // few right-hand sides: one warp per row (the 16 × 16 tiles would idle)
    switch (nrhs * 2 + (a_lo ? 1 : 0)) {
      case 2: launch_rows_df<1, false>(m, n, a_hi, a_lo, lda, xh, xl, nn, y, b, ldy, st); break;
      case 3: launch_rows_df<1, true>(m, n, a_hi, a_lo, lda, xh, xl, nn, y, b, ldy, st); break;
      case 4: launch_rows_df<2, false>(m, n, a_hi, a_lo, lda, xh, xl, nn, y, b, ldy, st); break;
      case 5: launch_rows_df<2, true>(m, n, a_hi, a_lo, lda, xh, xl, nn, y, b, ldy, st); break;
      case 6: launch_rows_df<3, false>(m, n, a_hi, a_lo, lda, xh, xl, nn, y, b, ldy, st); break;
      case 7: launch_rows_df<3, true>(m, n, a_hi, a_lo, lda, xh, xl, nn, y, b, ldy, st); break;
      case 8: launch_rows_df<4, false>(m, n, a_hi, a_lo, lda, xh, xl, nn, y, b, ldy, st); break;
      default: launch_rows_df<4, true>(m, n, a_hi, a_lo, lda, xh, xl, nn, y, b, ldy, st); break;
    }
    return check_launch("gemv_df");
  }
  if (mode == 0)
    return res ? launch_gemv16<0, 2>(m, n, a_hi, lda, nrhs, xh, nn, nullptr, y, b, ldy, st)
               : launch_gemv16<0, 1>(m, n, a_hi, lda, nrhs, xh, nn, nullptr, y, nullptr, ldy, st);
  if (a_lo)
    return res ? launch_df<true, 0, 2>(m, n, a_hi, a_lo, lda, nrhs, xh, xl, nn, nullptr, nullptr,
                                       y, b, ldy, st)
               : launch_df<true, 0, 1>(m, n, a_hi, a_lo, lda, nrhs, xh, xl, nn, nullptr, nullptr,
                                       y, nullptr, ldy, st);
  return res ? launch_df<false, 0, 2>(m, n, a_hi, nullptr, lda, nrhs, xh, xl, nn, nullptr, nullptr,
                                      y, b, ldy, st)
             : launch_df<false, 0, 1>(m, n, a_hi, nullptr, lda, nrhs, xh, xl, nn, nullptr, nullptr,
                                      y, nullptr, ldy, st);
}
