// FP64 symmetric rank-k products and the multi-CTA Cholesky of one large
// matrix.
//
// syrk_f64_kernel forms S = AᵀA (A k×n) or AAᵀ (A n×k) on the upper 64×64
// tiles of an n×n result, one CTA per tile (256 threads, 4×4 outputs each,
// A staged through shared memory in 16-deep slices).  Either as a Gram matrix
// (C = S, optionally mirrored into the lower triangle: the normal equations
// of lineax's Normal solver, lineax/_solver/normal.py:112-118) or as an update
// C -= S of the upper triangle, where every element continues its FMA chain
// from its stored value in k order (the Cholesky below has its own, 32 rows at
// a time).
//
// lxgb_potrf_f64 factors one n×n SPD matrix (A = UᵀU, upper) right-looking
// by 32-row block rows: the diagonal block and its block row in one sweep
// (potrf_row_kernel), the update of the next block row, and beside that next
// row the update of the rest.  Every element receives exactly the update chain of the
// single-CTA factorisation (k ascending, scaling by the pivot reciprocal), so
// both give the same bits.
#include "common.cuh"
#include "potrf.cuh"

namespace lxgb {

constexpr int kSyTile = 64;
constexpr int kSyK = 16;
constexpr int kPoNB = 32;       // block rows of the multi-CTA Cholesky
// Columns per CTA of the block-row kernel: 32 G.  G = 2 above kPoWide trailing
// columns, where the trailing update beside it wants the SMs (n = 1531: 24
// instead of 48 of them); G = 1 below, where the block row's own time counts
// (25 us against 30).  us for the factor with this line, with G = 1 and with G = 2
// throughout: n = 1000 1002, 997 and 1126, 1531 1999, 2120 and 2098, 3000 9367, 9663 and
// 9455, 8192 153400, 155200 and 153500.
constexpr int kPoWide = 1024;
// Unused dynamic shared memory that a block-row CTA reserves, so that no CTA
// of the trailing update running beside it (17 KB each) shares its SM.
constexpr int kPoReserve = 190 * 1024;

// Upper tile t (row-major over the triangle) of an nt×nt tile grid.
__device__ __forceinline__ void upper_tile(int t, int nt, int& ti, int& tj) {
  int rem = t, i = 0;
  while (rem >= nt - i) { rem -= nt - i; ++i; }
  ti = i;
  tj = i + rem;
}

// trans 0: S = AᵀA, element (kk, i) of the k×n operand at a[kk*lda + i];
// trans 1: S = AAᵀ, element (kk, i) at a[i*lda + kk].
// update 0: C = S (fill: also write C[j][i]); update 1: C -= S on j >= i.
__global__ void __launch_bounds__(256)
syrk_f64_kernel(int trans, int64_t n, int64_t k, const double* __restrict__ a, int64_t lda,
                int update, double* __restrict__ c, int64_t ldc, int fill) {
  __shared__ double as[kSyK][kSyTile + 1];
  __shared__ double bs[kSyK][kSyTile + 1];
  const int nt = (int)((n + kSyTile - 1) / kSyTile);
  int ti, tj;
  upper_tile(blockIdx.x, nt, ti, tj);
  const int64_t i0 = (int64_t)ti * kSyTile, j0 = (int64_t)tj * kSyTile;
  const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
  double acc[4][4];
#pragma unroll
  for (int r = 0; r < 4; ++r)
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const int64_t i = i0 + ty + 16 * r, j = j0 + tx + 16 * q;
      acc[r][q] = (update && i < n && j < n && j >= i) ? c[i * ldc + j] : 0.0;
    }
  for (int64_t k0 = 0; k0 < k; k0 += kSyK) {
#pragma unroll
    for (int e4 = 0; e4 < (kSyK * kSyTile) / 256; ++e4) {
      const int e = tid + 256 * e4;
      int kk, ii;
      if (trans == 0) { kk = e / kSyTile; ii = e % kSyTile; }
      else { ii = e / kSyK; kk = e % kSyK; }
      const int64_t gk = k0 + kk, gi = i0 + ii, gj = j0 + ii;
      double va = 0.0, vb = 0.0;
      if (gk < k) {
        if (trans == 0) {
          if (gi < n) va = a[gk * lda + gi];
          if (gj < n) vb = a[gk * lda + gj];
        } else {
          if (gi < n) va = a[gi * lda + gk];
          if (gj < n) vb = a[gj * lda + gk];
        }
      }
      as[kk][ii] = va;
      bs[kk][ii] = vb;
    }
    __syncthreads();
    const int kn = (int)((k - k0 < kSyK) ? (k - k0) : kSyK);
    for (int kk = 0; kk < kn; ++kk) {
      double ai[4], bj[4];
#pragma unroll
      for (int r = 0; r < 4; ++r) ai[r] = as[kk][ty + 16 * r];
#pragma unroll
      for (int q = 0; q < 4; ++q) bj[q] = bs[kk][tx + 16 * q];
#pragma unroll
      for (int r = 0; r < 4; ++r)
#pragma unroll
        for (int q = 0; q < 4; ++q)
          acc[r][q] = update ? fma(-ai[r], bj[q], acc[r][q]) : fma(ai[r], bj[q], acc[r][q]);
    }
    __syncthreads();
  }
#pragma unroll
  for (int r = 0; r < 4; ++r)
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const int64_t i = i0 + ty + 16 * r, j = j0 + tx + 16 * q;
      if (i < n && j < n && j >= i) {
        c[i * ldc + j] = acc[r][q];
        if (fill && !update && j > i) c[j * ldc + i] = acc[r][q];
      }
    }
}

// Block row [j0, j0+nb) of U: the diagonal block factored and U12 = U11⁻ᵀ A12
// formed in the same sweep.  A CTA takes the diagonal block and 32 G columns
// right of it; every CTA factors the block for itself.  Warp 0 runs the chain:
// in step k it has row k of the block in registers, forms the pivot's square
// root and reciprocal, scales the row, and after one barrier updates row k + 1
// for itself.  Six other warps hold the remaining rows in registers (row i with
// warp i mod 6, a lane per column of the block and one per column beside it),
// scale row k of the CTA's columns and update their rows; the owners of rows
// k + 1 and k + 2 pass on through shared memory what the next step reads.
// (Warp 4 shares warp 0's sub-partition and stays out of its way.)  What
// bounds it is warp 0's chain (the pivot's root and reciprocal, scaling, a barrier, FMA).
// Measured, n = 1531: 25 to 30 us a block row of 32 (27 to 31 with a square root
// and a division in the chain); a block
// row of 64 as a diagonal kernel (138 us) and a column-per-thread substitution
// (149 us) before.  The whole factorisation 8.4 to 2.0 ms.
// The operations on each element, and their order, are cta_potrf_upper's:
// row k scaled by 1 / sqrt(a_kk), then one FMA per later row, k ascending.
// Except for the last block, the factored block does not go back to its place: a CTA
// that starts late (more of them than SMs, or SMs taken by other streams) still
// reads the block unfactored.  CTA 0 keeps it below the diagonal, which no kernel
// of the sweep reads: off-diagonal entries transposed into the block's own lower
// triangle, its diagonal in the 32 entries of the row below the block;
// potrf_finish_kernel moves both.
constexpr int kPoOwners = 6;
constexpr int kPoRows = (kPoNB + kPoOwners - 1) / kPoOwners;

template <int G>
__global__ void __launch_bounds__(256)
potrf_row_kernel(int64_t n, double* __restrict__ a, int64_t lda, int64_t j0, int nb,
                 int32_t* __restrict__ info) {
  __shared__ double U[kPoNB][kPoNB + 1];   // finished rows of the block
  __shared__ double D[2][kPoNB];           // row k of the block as warp 0 takes it, by parity
  __shared__ double E[2][32 * G];          // row k beside it, not yet scaled
  __shared__ double s_r[2];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int64_t col = j0 + nb + (int64_t)blockIdx.x * (32 * G) + lane;  // and col + 32 h
  const int uw = (warp < 4) ? warp - 1 : warp - 2;   // owner 0..5 (warp 0: -1)
  const bool owner = warp != 0 && warp != 4;
  pdl_wait();
  // everything before is finished: the rest of the previous trailing update
  // may start beside this kernel
  pdl_trigger();
  double g[kPoRows], e[kPoRows][G];        // rows uw + 6 q: block, columns beside it
  double v = 0.0;
  if (owner) {
#pragma unroll
    for (int q = 0; q < kPoRows; ++q) {
      const int i = uw + kPoOwners * q;
      g[q] = (i < nb && lane >= i && lane < nb) ? a[(j0 + i) * lda + j0 + lane] : 0.0;
#pragma unroll
      for (int h = 0; h < G; ++h)
        e[q][h] = (i < nb && col + 32 * h < n) ? a[(j0 + i) * lda + col + 32 * h] : 0.0;
    }
    if (uw == 0) {
#pragma unroll
      for (int h = 0; h < G; ++h) E[0][lane + 32 * h] = e[0][h];
    }
    if (uw == 1) D[1][lane] = g[0];
  } else if (warp == 0) {
    v = (lane < nb) ? a[j0 * lda + j0 + lane] : 0.0;
  }
  int bad = 0;
  for (int k = 0; k < nb; ++k) {
    const int par = k & 1;
    double u = 0.0;
    if (warp == 0) {
      const double akk = __shfl_sync(0xffffffffu, v, k);
      if (!(akk > 0.0) && bad == 0) bad = k + 1;
      double d, r;
      potrf_pivot(akk, d, r);
      u = (lane > k) ? v * r : (lane == k ? d : 0.0);
      U[k][lane] = u;
      if (lane == 0) s_r[par] = r;
    }
    __syncthreads();
    if (warp == 0) {
      const double uk1 = __shfl_sync(0xffffffffu, u, min(k + 1, kPoNB - 1));
      v = fma(-uk1, u, D[par ^ 1][lane]);              // row k + 1
    } else if (owner) {
      const double ul = U[k][lane];
      double x[G];
#pragma unroll
      for (int h = 0; h < G; ++h) {
        x[h] = E[par][lane + 32 * h] * s_r[par];
        if (uw == k % kPoOwners && col + 32 * h < n) a[(j0 + k) * lda + col + 32 * h] = x[h];
      }
#pragma unroll
      for (int q = 0; q < kPoRows; ++q) {
        const int i = uw + kPoOwners * q;
        if (i > k && i < nb) {                         // uniform over the warp
          const double ui = U[k][i];
#pragma unroll
          for (int h = 0; h < G; ++h) {
            e[q][h] = fma(-ui, x[h], e[q][h]);
            if (i == k + 1) E[par ^ 1][lane + 32 * h] = e[q][h];
          }
          if (i != k + 1) {
            g[q] = fma(-ui, ul, g[q]);
          }
          if (i == k + 2) D[par][lane] = g[q];
        }
      }
    }
  }
  if (blockIdx.x == 0) {
    __syncthreads();
    if (j0 + nb == n) {                                // no CTA beside this one
      for (int t = tid; t < nb * nb; t += 256) {
        const int i = t / nb, j = t % nb;
        if (j >= i) a[(j0 + i) * lda + j0 + j] = U[i][j];
      }
    } else {                                           // (nb is kPoNB)
      for (int t = tid; t < kPoNB * kPoNB; t += 256) {
        const int i = t % kPoNB, j = t / kPoNB;
        if (j > i) a[(j0 + j) * lda + j0 + i] = U[i][j];
      }
      if (tid < kPoNB) a[(j0 + kPoNB) * lda + j0 + tid] = U[tid][tid];
    }
    if (tid == 0 && bad != 0 && info[0] == 0) info[0] = (int32_t)(j0 + bad);
  }
}

// The next block row's share of the trailing update, ahead of the rest: rows
// [s, s+32), s = j0 + nb, columns j >= i, a_ij -= sum_k u_ki u_kj.  32x8 tile
// per CTA (the critical path: as many SMs as there are tiles).
__global__ void __launch_bounds__(128)
potrf_next_row_kernel(int64_t n, double* __restrict__ a, int64_t lda, int64_t j0, int nb) {
  __shared__ double Ui[kPoNB][kPoNB + 1];
  __shared__ double Uj[kPoNB][8];
  const int64_t s = j0 + nb;
  const int64_t c0 = s + (int64_t)blockIdx.x * 8;
  const int tid = threadIdx.x;
  const int tx = tid & 7, ty = tid >> 3;
  const int64_t j = c0 + tx;
  pdl_wait();
  double acc[2];
#pragma unroll
  for (int r = 0; r < 2; ++r) {
    const int64_t i = s + ty + 16 * r;
    acc[r] = (i < n && j < n && j >= i) ? a[i * lda + j] : 0.0;
  }
#pragma unroll
  for (int e = tid; e < kPoNB * kPoNB; e += 128) {
    const int k = e / kPoNB, i = e % kPoNB;
    Ui[k][i] = (k < nb && s + i < n) ? a[(j0 + k) * lda + s + i] : 0.0;
  }
#pragma unroll
  for (int e = tid; e < kPoNB * 8; e += 128) {
    const int k = e / 8, c = e % 8;
    Uj[k][c] = (k < nb && c0 + c < n) ? a[(j0 + k) * lda + c0 + c] : 0.0;
  }
  __syncthreads();
#pragma unroll 8
  for (int k = 0; k < nb; ++k) {
    const double uj = Uj[k][tx];
#pragma unroll
    for (int r = 0; r < 2; ++r) acc[r] = fma(-Ui[k][ty + 16 * r], uj, acc[r]);
  }
  pdl_trigger();
#pragma unroll
  for (int r = 0; r < 2; ++r) {
    const int64_t i = s + ty + 16 * r;
    if (i < n && j < n && j >= i) a[i * lda + j] = acc[r];
  }
}

// The rest of the trailing update: rows and columns from s = j0 + nb + 32 on,
// upper 32x32 tiles, 2x4 outputs per thread.  Runs beside the next block row:
// it reads at once what was finished before that kernel (through L2), touches
// none of its elements, and waits for it only before it ends (as the LU's
// trailing update does).
__global__ void __launch_bounds__(128)
potrf_trailing_kernel(int64_t n, double* a, int64_t lda, int64_t j0, int nb, int64_t s) {
  __shared__ double Ui[kPoNB][kPoNB + 1];
  __shared__ double Uj[kPoNB][kPoNB + 2];
  const int nt = (int)((n - s + kPoNB - 1) / kPoNB);
  int ti, tj;
  upper_tile(blockIdx.x, nt, ti, tj);
  const int64_t i0 = s + (int64_t)ti * kPoNB, c0 = s + (int64_t)tj * kPoNB;
  const int tid = threadIdx.x, tx = tid & 7, ty = tid >> 3;
  double acc[2][4];
#pragma unroll
  for (int r = 0; r < 2; ++r)
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const int64_t i = i0 + ty + 16 * r, j = c0 + tx + 8 * q;
      acc[r][q] = (i < n && j < n && j >= i) ? __ldcg(a + i * lda + j) : 0.0;
    }
#pragma unroll
  for (int e = tid; e < kPoNB * kPoNB; e += 128) {
    const int k = e / kPoNB, i = e % kPoNB;
    Ui[k][i] = (k < nb && i0 + i < n) ? __ldcg(a + (j0 + k) * lda + i0 + i) : 0.0;
    Uj[k][i] = (k < nb && c0 + i < n) ? __ldcg(a + (j0 + k) * lda + c0 + i) : 0.0;
  }
  __syncthreads();
#pragma unroll 8
  for (int k = 0; k < nb; ++k) {
    double ui[2], uj[4];
#pragma unroll
    for (int r = 0; r < 2; ++r) ui[r] = Ui[k][ty + 16 * r];
#pragma unroll
    for (int q = 0; q < 4; ++q) uj[q] = Uj[k][tx + 8 * q];
#pragma unroll
    for (int r = 0; r < 2; ++r)
#pragma unroll
      for (int q = 0; q < 4; ++q) acc[r][q] = fma(-ui[r], uj[q], acc[r][q]);
  }
#pragma unroll
  for (int r = 0; r < 2; ++r)
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const int64_t i = i0 + ty + 16 * r, j = c0 + tx + 8 * q;
      if (i < n && j < n && j >= i) a[i * lda + j] = acc[r][q];
    }
  pdl_wait();
}

// The block columns of the finished factor: the diagonal block that
// potrf_row_kernel left below the diagonal into its place (but for the last block,
// which is there), and zeros below the diagonal.  CTA (b, y): block b, rows
// [kPoFinish y, kPoFinish (y + 1)) below it; y = 0 also the block.
constexpr int kPoFinish = 256;

__global__ void __launch_bounds__(256)
potrf_finish_kernel(int64_t n, double* __restrict__ a, int64_t lda) {
  __shared__ double U[kPoNB][kPoNB + 1];
  const int64_t j0 = (int64_t)blockIdx.x * kPoNB;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int64_t s = j0 + kPoNB;                        // first row below the block
  if (blockIdx.y == 0) {
    const bool moved = s < n;
    if (moved) {
      for (int i = warp; i < kPoNB; i += 8)
        U[i][lane] = (lane < i) ? a[(j0 + i) * lda + j0 + lane]
                                : (lane == i ? a[s * lda + j0 + lane] : 0.0);
      __syncthreads();
    }
    for (int i = warp; i < kPoNB && j0 + i < n; i += 8) {
      double* row = a + (j0 + i) * lda + j0;
      if (lane < i) row[lane] = 0.0;
      else if (moved) row[lane] = U[lane][i];
    }
    __syncthreads();                                   // the row below was read above
  }
  const int64_t lo = s + (int64_t)blockIdx.y * kPoFinish;
  for (int64_t i = lo + warp; i < n && i < lo + kPoFinish; i += 8) a[i * lda + j0 + lane] = 0.0;
}

__global__ void set_info_kernel(int32_t* info) { info[0] = 0; }

static int syrk_launch(int trans, int64_t n, int64_t k, const double* a, int64_t lda, int update,
                       double* c, int64_t ldc, int fill, cudaStream_t st) {
  const int64_t nt = (n + kSyTile - 1) / kSyTile;
  const int64_t tiles = nt * (nt + 1) / 2;
  LXGB_REQUIRE(tiles < (1LL << 31), "syrk: n too large");
  syrk_f64_kernel<<<(unsigned)tiles, 256, 0, st>>>(trans, n, k, a, lda, update, c, ldc, fill);
  return check_launch("syrk_f64");
}

}  // namespace lxgb

using namespace lxgb;

extern "C" int lxgb_syrk_f64(int32_t trans, int64_t n, int64_t k, const double* a, int64_t lda,
                             int32_t update, double* c, int64_t ldc, int32_t fill, void* stream) {
  LXGB_REQUIRE(n >= 0 && k >= 0, "syrk: negative size");
  LXGB_REQUIRE(trans == 0 || trans == 1, "syrk: trans must be 0 or 1");
  LXGB_REQUIRE(!(update && fill), "syrk: fill is for the Gram form (update == 0)");
  if (n == 0) return LXGB_SUCCESSFUL;
  LXGB_REQUIRE(c && (k == 0 || a), "syrk: null pointer");
  LXGB_REQUIRE(ldc >= n && lda >= (trans == 0 ? n : k), "syrk: leading dimension too small");
  return syrk_launch(trans, n, k, a, lda, update, c, ldc, fill, as_stream(stream));
}

extern "C" int lxgb_potrf_f64(int64_t n, double* a, int64_t lda, int32_t* info, void* stream) {
  LXGB_REQUIRE(n >= 0, "potrf: negative size");
  LXGB_REQUIRE(info, "potrf: null info");
  cudaStream_t st = as_stream(stream);
  set_info_kernel<<<1, 1, 0, st>>>(info);
  if (n == 0) return check_launch("potrf_f64");
  LXGB_REQUIRE(a && lda >= n, "potrf: null pointer or lda < n");
  for (const void* fn : {reinterpret_cast<const void*>(potrf_row_kernel<1>),
                         reinterpret_cast<const void*>(potrf_row_kernel<2>)})
    LXGB_CUDA_TRY(ensure_dynamic_smem(fn, kPoReserve), "potrf: set smem");
  LXGB_REQUIRE(n < (1LL << 31) - 64, "potrf: n too large");
  // per block row: the row itself, its update of the next row, and (beside the
  // next row) of everything after that
  for (int64_t j0 = 0; j0 < n; j0 += kPoNB) {
    const int nb = (int)((n - j0 < kPoNB) ? (n - j0) : kPoNB);
    const int64_t rest = n - j0 - nb;
    const int cols = rest > kPoWide ? 64 : 32;
    const int64_t ctas = rest > 0 ? (rest + cols - 1) / cols : 1;
    LXGB_CUDA_TRY(launch_pdl(cols == 64 ? potrf_row_kernel<2> : potrf_row_kernel<1>,
                             dim3((unsigned)ctas), dim3(256), kPoReserve, st, 1, n, a, lda, j0, nb,
                             info),
                  "potrf: block row launch");
    // the previous row's trailing update, released once this row's CTAs run
    if (j0 > 0 && rest > 0) {
      const int64_t nt = (rest + kPoNB - 1) / kPoNB;
      LXGB_REQUIRE(nt * (nt + 1) / 2 < (1LL << 31), "potrf: n too large");
      LXGB_CUDA_TRY(launch_pdl(potrf_trailing_kernel, dim3((unsigned)(nt * (nt + 1) / 2)),
                               dim3(128), 0, st, 1, n, a, lda, j0 - kPoNB, (int)kPoNB, j0 + nb),
                    "potrf: trailing update launch");
    }
    if (rest > 0)
      LXGB_CUDA_TRY(launch_pdl(potrf_next_row_kernel, dim3((unsigned)((rest + 7) / 8)), dim3(128),
                               0, st, 1, n, a, lda, j0, nb),
                    "potrf: next row update launch");
  }
  const int64_t blocks = (n + kPoNB - 1) / kPoNB;
  const int64_t below = n > kPoNB ? (n - kPoNB + kPoFinish - 1) / kPoFinish : 1;
  LXGB_REQUIRE(below <= 65535, "potrf: n too large");
  potrf_finish_kernel<<<dim3((unsigned)blocks, (unsigned)below), 256, 0, st>>>(n, a, lda);
  return check_launch("potrf_f64");
}
