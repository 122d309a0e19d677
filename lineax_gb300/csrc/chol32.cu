// FP32 Cholesky of one large SPD matrix with tensor-core updates, for
// mixed-precision refinement (the serving route of Cholesky requests above
// the ragged kernel's order limit):
//
//   lxgb_potrf_f32_tc  — A = L Lᵀ in FP32, right-looking by 64-column panels:
//     the 64×64 diagonal block and the panel below it L21 = A21 L_jj⁻ᵀ in one
//     launch (FP32 on the CUDA cores), and the trailing update A22 -= L21 L21ᵀ
//     (lower-triangle tiles only) as a tcgen05 GEMM with 3xTF32 products
//     (FP32-level accuracy).  A is read from its upper triangle, as
//     lineax's Cholesky reads it (cho_factor(lower=False),
//     lineax/_solver/cholesky.py:60): L = Uᵀ.
//   lxgb_chol32_to_lu32 — the factor in the unit-lower / upper form of the
//     mixed LU (L' = L D⁻¹, U' = D Lᵀ, D = diag(L), no interchanges), so the
//     GMRES-IR machinery of the mixed LU applies unchanged.
//   lxgb_chol32_uinv    — U'⁻¹ = L'⁻ᵀ D⁻² from L'⁻¹: the second triangular
//     inverse by a transposing copy instead of a second substitution.
#include "common.cuh"
#include "tc_gemm.cuh"

namespace lxgb {

constexpr int kC32NB = 64;

// l[i][j] = fl32(a[j][i]) for j <= i (A's upper triangle, transposed), 0
// above the diagonal.  32×32 tiles through shared memory: coalesced reads of
// a's rows and writes of l's rows.
__global__ void c32_lower_from_upper_kernel(int64_t n, const double* __restrict__ a,
                                            float* __restrict__ l) {
  __shared__ float tile[32][33];
  const int64_t bi = (int64_t)blockIdx.y * 32, bj = (int64_t)blockIdx.x * 32;  // tile of l
  // read a[bj + r][bi + c] (a row segment) into tile[r][c]
  for (int r = threadIdx.y; r < 32; r += blockDim.y) {
    const int64_t ar = bj + r, ac = bi + threadIdx.x;
    tile[r][threadIdx.x] = (ar < n && ac < n) ? __double2float_rn(a[ar * n + ac]) : 0.0f;
  }
  __syncthreads();
  for (int r = threadIdx.y; r < 32; r += blockDim.y) {
    const int64_t li = bi + r, lj = bj + threadIdx.x;
    if (li < n && lj < n) l[li * n + lj] = (lj <= li) ? tile[threadIdx.x][r] : 0.0f;
  }
}

// One block column: the 64×64 diagonal block at (j0, j0) of l (nb×nb at the
// end) factored, and the rows below it L21 = A21 L_jj⁻ᵀ, 128 per CTA, one per
// thread.  Every CTA factors the block for itself (its own copy; CTA 0 stores it
// in diag, from where c32_store_diag_kernel takes it at the end — a CTA that
// starts late still reads the block unfactored).
//  * Factor: row tid & 63 in the registers of two threads, which hold the even
//    and the odd columns.  Columns in registers are kept shifted, element 0 being
//    the next column of its parity, so one loop body serves all 64: the owners
//    publish the raw column, each takes the root, the owners divide, and all
//    apply the rank-1 update.  A pivot that is not positive counts as 1; the
//    first is recorded in *info (1-based, global).
//  * Rows: 16 columns at a time in registers, as one body for the product with a
//    16×16 block and one for the triangle.  L21 goes back into l and, split into
//    TF32-exact hi and lo parts, into ph / pl (row stride 64).
// Bound by the two chains of 64 steps (a root, a division and two barriers; a
// division).  Measured per block column at n = 2048, with the update: 44 us (102
// with the block in one CTA and the panel in a launch of its own).
constexpr int kC32Threads = 128;
constexpr int kC32T = 16;
constexpr int kC32TLd = kC32NB + 4;
constexpr int kC32XLd = kC32NB + 1;
constexpr int kC32Smem = (kC32NB * kC32TLd + kC32Threads * kC32XLd) * (int)sizeof(float);

__global__ void __launch_bounds__(kC32Threads)
c32_row_kernel(int64_t n, int64_t j0, int nb, int m2, float* __restrict__ l,
               float* __restrict__ diag, float* __restrict__ ph, float* __restrict__ pl,
               int32_t* __restrict__ info) {
  extern __shared__ __align__(16) float c32_smem[];
  float (*Tt)[kC32TLd] = reinterpret_cast<float (*)[kC32TLd]>(c32_smem);  // Tt[k][i] = L[i][k]
  float (*X)[kC32XLd] = reinterpret_cast<float (*)[kC32XLd]>(c32_smem + kC32NB * kC32TLd);
  // the raw and the scaled column, alternating with the column's parity; the
  // scaled one by parity of the row, from the current pair of columns on
  __shared__ __align__(16) float raw[2][kC32NB], col[2][2][kC32NB / 2];
  constexpr int kLoads = 32;
  const int tid = threadIdx.x, i = tid & (kC32NB - 1), h = tid >> 6;
  const int64_t rbase = (int64_t)blockIdx.x * kC32Threads;  // first row below the block
  {
    float v[kLoads];
#pragma unroll
    for (int u = 0; u < kLoads; ++u) {
      const int e = tid + u * kC32Threads, r = e / kC32NB, c = e % kC32NB;
      v[u] = (r < nb && c <= r) ? l[(j0 + r) * n + j0 + c] : (r == c ? 1.0f : 0.0f);
    }
#pragma unroll
    for (int u = 0; u < kLoads; ++u) {
      const int e = tid + u * kC32Threads;
      X[e / kC32NB][e % kC32NB] = v[u];
    }
  }
  __syncthreads();
  float r[kC32NB / 2];
#pragma unroll
  for (int j = 0; j < kC32NB / 2; ++j) r[j] = X[i][2 * j + h];
  // the rows below, on their way while the block is factored
  float a[kLoads];
#pragma unroll
  for (int u = 0; u < kLoads; ++u) {
    const int e = tid + u * kC32Threads, rr = e / kC32NB, c = e % kC32NB;
    a[u] = (rbase + rr < m2) ? l[(j0 + kC32NB + rbase + rr) * n + j0 + c] : 0.0f;
  }
  int bad = 0;
#pragma unroll 1
  for (int kk = 0; kk < kC32NB / 2; ++kk) {
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      const int k = 2 * kk + q;
      if (h == q) raw[q][i] = r[0];
      __syncthreads();
      float d = raw[q][k];
      if (!(d > 0.0f)) {
        if (bad == 0) bad = k + 1;
        d = 1.0f;
      }
      const float s = sqrtf(d);
      if (h == q && i >= k) {
        const float v = (i == k) ? s : r[0] / s;
        Tt[k][i] = v;
        col[q][i & 1][(i >> 1) - kk] = v;
      }
      __syncthreads();
      const float li = (i > k) ? col[q][i & 1][(i >> 1) - kk] : 0.0f;
      const float4* cq = reinterpret_cast<const float4*>(col[q][h]);
#pragma unroll
      for (int j4 = 0; j4 < kC32NB / 8; ++j4) {
        const float4 t = cq[j4];
        const float tv[4] = {t.x, t.y, t.z, t.w};
#pragma unroll
        for (int w = 0; w < 4; ++w) {
          const int j = 4 * j4 + w;
          // columns 2 (kk + j) + h > k; rows above the diagonal hold nothing
          if (q == 0) {
            if (j > 0 || h == 1) r[j] = (i > k) ? fmaf(-li, tv[w], r[j]) : 0.0f;
          } else if (j > 0) {
            r[j - 1] = (i > k) ? fmaf(-li, tv[w], r[j]) : 0.0f;
          }
        }
      }
    }
  }
  __syncthreads();
  if (blockIdx.x == 0) {
    float* dst = diag + j0 * kC32NB;
    for (int e = tid; e < kC32NB * kC32NB; e += kC32Threads) {
      const int rr = e / kC32NB, c = e % kC32NB;
      if (rr < nb && c <= rr) dst[e] = Tt[c][rr];
    }
    if (tid == 0 && bad) atomicCAS(reinterpret_cast<int*>(info), 0, (int)(j0 + bad));
  }
  if (m2 <= 0) return;
  // (the block's copy in X was read before the first barrier of the factor)
#pragma unroll
  for (int g = 0; g < 2; ++g) {
    if (g == 1) {
#pragma unroll
      for (int u = 0; u < kLoads; ++u) {
        const int e = tid + (u + kLoads) * kC32Threads, rr = e / kC32NB, c = e % kC32NB;
        a[u] = (rbase + rr < m2) ? l[(j0 + kC32NB + rbase + rr) * n + j0 + c] : 0.0f;
      }
    }
#pragma unroll
    for (int u = 0; u < kLoads; ++u) {
      const int e = tid + (u + g * kLoads) * kC32Threads;
      X[e / kC32NB][e % kC32NB] = a[u];
    }
  }
  __syncthreads();
#pragma unroll 1
  for (int bi = 0; bi < kC32NB / kC32T; ++bi) {
    const int i0 = bi * kC32T;
    float x[kC32T];
#pragma unroll
    for (int c = 0; c < kC32T; ++c) x[c] = X[tid][i0 + c];
#pragma unroll 1
    for (int k0 = 0; k0 < i0; k0 += kC32T) {
#pragma unroll
      for (int k = 0; k < kC32T; ++k) {
        const float xk = X[tid][k0 + k];
#pragma unroll
        for (int c4 = 0; c4 < kC32T / 4; ++c4) {
          const float4 t = *reinterpret_cast<const float4*>(&Tt[k0 + k][i0 + 4 * c4]);
          x[4 * c4 + 0] = fmaf(-xk, t.x, x[4 * c4 + 0]);
          x[4 * c4 + 1] = fmaf(-xk, t.y, x[4 * c4 + 1]);
          x[4 * c4 + 2] = fmaf(-xk, t.z, x[4 * c4 + 2]);
          x[4 * c4 + 3] = fmaf(-xk, t.w, x[4 * c4 + 3]);
        }
      }
    }
#pragma unroll
    for (int k = 0; k < kC32T; ++k) {
      x[k] = x[k] / Tt[i0 + k][i0 + k];
#pragma unroll
      for (int c = k + 1; c < kC32T; ++c) x[c] = fmaf(-x[k], Tt[i0 + k][i0 + c], x[c]);
    }
#pragma unroll
    for (int c = 0; c < kC32T; ++c) X[tid][i0 + c] = x[c];
  }
  __syncthreads();
#pragma unroll 16
  for (int u = 0; u < 2 * kLoads; ++u) {
    const int e = tid + u * kC32Threads, rr = e / kC32NB, c = e % kC32NB;
    const int64_t pr = rbase + rr;
    if (pr < m2) {
      const float x = X[rr][c];
      const float hi = __uint_as_float(__float_as_uint(x) & 0xFFFFE000u);
      l[(j0 + kC32NB + pr) * n + j0 + c] = x;
      ph[pr * kC32NB + c] = hi;
      pl[pr * kC32NB + c] = x - hi;
    }
  }
}

// The factored diagonal blocks (64×64 each, lower triangles) into l.
__global__ void c32_store_diag_kernel(int64_t n, const float* __restrict__ diag,
                                      float* __restrict__ l) {
  const int64_t j0 = (int64_t)blockIdx.x * kC32NB;
  for (int e = threadIdx.x; e < kC32NB * kC32NB; e += blockDim.x) {
    const int64_t r = e / kC32NB, c = e % kC32NB;
    if (c <= r && j0 + r < n) l[(j0 + r) * n + j0 + c] = diag[j0 * kC32NB + e];
  }
}

// The mixed-LU form of a Cholesky factor: lu[i][j] = L[i][j] / L[j][j] for
// j < i, lu[i][j] = L[i][i] L[j][i] for j >= i (U' = D Lᵀ).  32×32 tiles:
// tile (bi, bj) of lu needs tile (bj, bi) of L (transposed) above the
// diagonal and tile (bi, bj) below it; the diagonal values come from global
// memory.
__global__ void c32_to_lu_kernel(int64_t n, const float* __restrict__ l, float* __restrict__ lu) {
  __shared__ float tile[32][33];
  const int64_t bi = (int64_t)blockIdx.y * 32, bj = (int64_t)blockIdx.x * 32;
  for (int r = threadIdx.y; r < 32; r += blockDim.y) {
    const int64_t tr = bj + r, tc = bi + threadIdx.x;   // L[bj + r][bi + x]
    tile[r][threadIdx.x] = (tr < n && tc < n) ? l[tr * n + tc] : 0.0f;
  }
  __syncthreads();
  for (int r = threadIdx.y; r < 32; r += blockDim.y) {
    const int64_t i = bi + r, j = bj + threadIdx.x;
    if (i >= n || j >= n) continue;
    float v;
    if (j < i)
      v = l[i * n + j] / l[j * n + j];
    else
      v = l[i * n + i] * tile[threadIdx.x][r];          // L[i][i] * L[j][i]
    lu[i * n + j] = v;
  }
}

// uinv[i][j] = linv[j][i] / lu[j][j] for j >= i, 0 below the diagonal.
__global__ void c32_uinv_kernel(int64_t n, const float* __restrict__ lu,
                                const float* __restrict__ linv, float* __restrict__ uinv) {
  __shared__ float tile[32][33];
  const int64_t bi = (int64_t)blockIdx.y * 32, bj = (int64_t)blockIdx.x * 32;
  for (int r = threadIdx.y; r < 32; r += blockDim.y) {
    const int64_t tr = bj + r, tc = bi + threadIdx.x;   // linv[bj + r][bi + x]
    tile[r][threadIdx.x] = (tr < n && tc < n) ? linv[tr * n + tc] : 0.0f;
  }
  __syncthreads();
  for (int r = threadIdx.y; r < 32; r += blockDim.y) {
    const int64_t i = bi + r, j = bj + threadIdx.x;
    if (i >= n || j >= n) continue;
    uinv[i * n + j] = (j >= i) ? tile[threadIdx.x][r] / lu[j * n + j] : 0.0f;
  }
}

__global__ void c32_iota_kernel(int64_t n, int32_t* __restrict__ piv) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x)
    piv[i] = (int32_t)i;
}

static dim3 c32_tiles(int64_t n) {
  return dim3((unsigned)((n + 31) / 32), (unsigned)((n + 31) / 32));
}

}  // namespace lxgb

using namespace lxgb;

extern "C" int64_t lxgb_potrf_f32_tc_workspace_size(int64_t n) {
  const int64_t panel = (n > 0 ? n : 1) * kC32NB * 4;
  // two panels and the factored diagonal blocks
  const int64_t diag = (panel / 4 + kC32NB * kC32NB) * 4;
  return 256 + 2 * ((panel + 255) / 256 * 256) + (diag + 255) / 256 * 256;
}

extern "C" int lxgb_potrf_f32_tc(int64_t n, const double* a, float* l, int32_t* info,
                                 int32_t* err, void* work, int64_t work_bytes, void* stream) {
  LXGB_REQUIRE(n >= 0, "potrf_f32_tc: negative size");
  if (n == 0) return LXGB_SUCCESSFUL;
  LXGB_REQUIRE(a && l && info && err && work, "potrf_f32_tc: null pointer");
  LXGB_REQUIRE(n < 32768, "potrf_f32_tc: n above 32767");
  LXGB_REQUIRE((n % 4) == 0, "potrf_f32_tc: n must be a multiple of 4 (16-byte TMA rows)");
  LXGB_REQUIRE((((uintptr_t)l) & 15) == 0 && (((uintptr_t)work) & 255) == 0,
               "potrf_f32_tc: l must be 16-byte and work 256-byte aligned");
  if (work_bytes < lxgb_potrf_f32_tc_workspace_size(n)) {
    set_last_error("potrf_f32_tc: workspace too small");
    return LXGB_WORKSPACE_TOO_SMALL;
  }
  cudaStream_t st = as_stream(stream);
  LXGB_CUDA_TRY(cudaMemsetAsync(info, 0, sizeof(int32_t), st), "potrf_f32_tc: clear info");
  c32_lower_from_upper_kernel<<<c32_tiles(n), dim3(32, 8), 0, st>>>(n, a, l);
  const int64_t panel = ((n * kC32NB * 4) + 255) / 256 * 256;
  char* wb = reinterpret_cast<char*>(work) + 256;
  float* ph = reinterpret_cast<float*>(wb);
  float* pl = reinterpret_cast<float*>(wb + panel);
  float* diag = reinterpret_cast<float*>(wb + 2 * panel);
  LXGB_CUDA_TRY(ensure_dynamic_smem(reinterpret_cast<const void*>(c32_row_kernel), kC32Smem),
                "potrf_f32_tc: set smem");
  for (int64_t j0 = 0; j0 < n; j0 += kC32NB) {
    const int nb = (int)(n - j0 < kC32NB ? n - j0 : kC32NB);
    const int m2 = (int)(n - j0 - nb);   // only the last block is narrower than 64
    const int ctas = m2 > 0 ? (m2 + kC32Threads - 1) / kC32Threads : 1;
    c32_row_kernel<<<(unsigned)ctas, kC32Threads, kC32Smem, st>>>(n, j0, nb, m2, l, diag, ph, pl,
                                                                  info);
    if (m2 <= 0) break;
    // A22 -= L21 L21ᵀ (3xTF32) on the tiles holding A22's lower triangle
    const int64_t r0 = j0 + kC32NB;
    const int rc = gemm_tf32_nt_split_lower(m2, kC32NB, ph, pl, kC32NB, l + r0 * n + r0, n,
                                            -1.0f, 1.0f, err, st);
    if (rc) return rc;
  }
  c32_store_diag_kernel<<<(unsigned)((n + kC32NB - 1) / kC32NB), 256, 0, st>>>(n, diag, l);
  return check_launch("potrf_f32_tc");
}

extern "C" int lxgb_chol32_to_lu32(int64_t n, const float* l, float* lu, int32_t* piv,
                                   void* stream) {
  LXGB_REQUIRE(n >= 0, "chol32_to_lu32: negative size");
  if (n == 0) return LXGB_SUCCESSFUL;
  LXGB_REQUIRE(l && lu && piv && l != lu, "chol32_to_lu32: null or aliased pointer");
  cudaStream_t st = as_stream(stream);
  c32_to_lu_kernel<<<c32_tiles(n), dim3(32, 8), 0, st>>>(n, l, lu);
  c32_iota_kernel<<<(unsigned)((n + 255) / 256 < 1024 ? (n + 255) / 256 : 1024), 256, 0, st>>>(
      n, piv);
  return check_launch("chol32_to_lu32");
}

extern "C" int lxgb_chol32_uinv(int64_t n, const float* lu, const float* linv, float* uinv,
                                void* stream) {
  LXGB_REQUIRE(n >= 0, "chol32_uinv: negative size");
  if (n == 0) return LXGB_SUCCESSFUL;
  LXGB_REQUIRE(lu && linv && uinv && linv != uinv, "chol32_uinv: null or aliased pointer");
  c32_uinv_kernel<<<c32_tiles(n), dim3(32, 8), 0, as_stream(stream)>>>(n, lu, linv, uinv);
  return check_launch("chol32_uinv");
}
