// Mixed-precision LU: FP32 storage, partial pivoting, trailing updates on the
// tcgen05 tensor cores (TF32 products, FP32 accumulation), and the matching
// FP32 solve used as the preconditioner of FP64 GMRES-IR.
//
// Right-looking blocked LU with 64-column panels:
//   panel_getf2_cluster_reg_kernel — getf2 on the panel with each row in
//                            one thread's registers across a thread-block
//                            cluster (up to 16 CTAs × 512 rows); pivot
//                            search and pivot row exchanged through
//                            distributed shared memory.
//   panel_getf2_cluster_kernel — the same with the panel in the cluster's
//                            shared memory (taller panels); and
//                            panel_getf2_f32_kernel (one CTA, panel in global
//                            memory) for panels too tall for either.
//   lu32_block_row         — the panel's row interchanges on the other columns,
//                            U12 = L11^{-1} A12 in place, and the operands of
//                            the update as K-major buffers (ir.cu)
//   gemm_tf32_nt           — A22 -= L21 U12 on the tensor cores
#include <cooperative_groups.h>
#include <cuda_bf16.h>
#include <float.h>
#include <limits.h>

#include <map>
#include <mutex>
#include <tuple>

#include "common.cuh"
#include "tc_gemm.cuh"
#include "tri.cuh"

namespace lxgb {

constexpr int kLu32NB = 64;
constexpr int kLu32PanelThreads = 1024;

__device__ __forceinline__ void warp_argmax_first_f(float& v, int& idx) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const float ov = __shfl_xor_sync(0xffffffffu, v, o);
    const int oi = __shfl_xor_sync(0xffffffffu, idx, o);
    if (ov > v || (ov == v && oi < idx)) { v = ov; idx = oi; }
  }
}

__global__ void __launch_bounds__(kLu32PanelThreads)
panel_getf2_f32_kernel(int n, int j0, int nb, float* __restrict__ a, int32_t* __restrict__ piv,
                       int32_t* __restrict__ info) {
  __shared__ float s_v[32];
  __shared__ int s_i[32];
  __shared__ int s_p;
  __shared__ float s_akk, s_old;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int nwarps = blockDim.x >> 5;
  for (int k = j0; k < j0 + nb; ++k) {
    float v = -1.0f;
    int idx = INT_MAX;
    for (int i = k + tid; i < n; i += blockDim.x) {
      const float x = fabsf(a[(int64_t)i * n + k]);
      if (x > v) { v = x; idx = i; }
    }
    warp_argmax_first_f(v, idx);
    if (lane == 0) { s_v[warp] = v; s_i[warp] = idx; }
    __syncthreads();
    if (warp == 0) {
      v = lane < nwarps ? s_v[lane] : -1.0f;
      idx = lane < nwarps ? s_i[lane] : INT_MAX;
      warp_argmax_first_f(v, idx);
      if (lane == 0) {
        if (idx == INT_MAX) idx = k;
        s_p = idx;
        s_akk = a[(int64_t)idx * n + k];
        s_old = a[(int64_t)k * n + k];
        piv[k] = idx;
        if (s_akk == 0.0f && *info == 0) *info = k + 1;
      }
    }
    __syncthreads();
    const int p = s_p;
    const float akk = s_akk;
    if (akk != 0.0f) {
      if (p != k) {
        for (int j = j0 + tid; j < j0 + nb; j += blockDim.x) {
          if (j == k) continue;
          const float t = a[(int64_t)k * n + j];
          a[(int64_t)k * n + j] = a[(int64_t)p * n + j];
          a[(int64_t)p * n + j] = t;
        }
      }
      const float r = 1.0f / akk;
      if (tid == 0) a[(int64_t)k * n + k] = akk;
      for (int i = k + 1 + tid; i < n; i += blockDim.x) {
        const float x = (i == p) ? s_old : a[(int64_t)i * n + k];
        a[(int64_t)i * n + k] = x * r;
      }
    }
    __syncthreads();
    const int w = j0 + nb - (k + 1);
    if (w > 0) {
      // rows i > k: one warp per row, lanes along the remaining panel columns
      for (int i = k + 1 + warp; i < n; i += nwarps) {
        const float l = a[(int64_t)i * n + k];
        for (int jj = lane; jj < w; jj += 32) {
          const int j = k + 1 + jj;
          a[(int64_t)i * n + j] = fmaf(-l, a[(int64_t)k * n + j], a[(int64_t)i * n + j]);
        }
      }
    }
    __syncthreads();
  }
}

namespace cg = cooperative_groups;

constexpr int kPanelCluThreads = 512;
constexpr int kPanelLd = kLu32NB + 1;  // padded row: column reads are conflict-free
constexpr int kPanelCluMax = 16;
constexpr size_t kPanelCluSmemMax = 200 * 1024;

// getf2 on the m×nb panel at (j0, j0) (m = n - j0), rows split over the
// cluster's CTAs (rows_per_cta each) and kept in shared memory for the whole
// panel.  Per column: each CTA's first max |a| is published; after a cluster
// barrier every CTA reduces the candidates (same order everywhere: first row
// of max |a|, as isamax), copies the pivot row and row kk out of their owners'
// shared memory, and after a second barrier the owners swap them and every CTA
// scales and updates its own rows.  Candidates are double-buffered by column
// parity, so one barrier pair per column suffices.  Arithmetic matches
// panel_getf2_f32_kernel (reciprocal scaling, fmaf rank-1 updates).
__global__ void __launch_bounds__(kPanelCluThreads)
panel_getf2_cluster_kernel(int n, int j0, int nb, int rows_per_cta, float* __restrict__ a,
                           int32_t* __restrict__ piv, int32_t* __restrict__ info) {
  extern __shared__ float P[];
  __shared__ float cand_v[2];
  __shared__ int cand_i[2];
  __shared__ float rowp[kLu32NB], rowk[kLu32NB];
  __shared__ float s_wv[kPanelCluThreads / 32];
  __shared__ int s_wi[kPanelCluThreads / 32];
  __shared__ int s_p;
  cg::cluster_group cluster = cg::this_cluster();
  const int ncta = (int)cluster.num_blocks();
  const int rank = (int)cluster.block_rank();
  const int m = n - j0;
  const int R = rows_per_cta;
  const int r0 = rank * R;
  const int mloc = max(0, min(R, m - r0));
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int nwarps = blockDim.x >> 5;
  for (int e = tid; e < mloc * kLu32NB; e += blockDim.x) {
    const int i = e / kLu32NB, j = e % kLu32NB;
    P[i * kPanelLd + j] = (j < nb) ? a[(int64_t)(j0 + r0 + i) * n + j0 + j] : 0.0f;
  }
  __syncthreads();
  for (int kk = 0; kk < nb; ++kk) {
    const int par = kk & 1;
    float v = -1.0f;
    int idx = INT_MAX;
    for (int i = tid; i < mloc; i += blockDim.x) {
      if (r0 + i >= kk) {
        const float x = fabsf(P[i * kPanelLd + kk]);
        if (x > v) { v = x; idx = r0 + i; }
      }
    }
    warp_argmax_first_f(v, idx);
    if (lane == 0) { s_wv[warp] = v; s_wi[warp] = idx; }
    __syncthreads();
    if (warp == 0) {
      v = lane < nwarps ? s_wv[lane] : -1.0f;
      idx = lane < nwarps ? s_wi[lane] : INT_MAX;
      warp_argmax_first_f(v, idx);
      if (lane == 0) { cand_v[par] = v; cand_i[par] = idx; }
    }
    cluster.sync();
    if (warp == 0) {
      float cv = -1.0f;
      int ci = INT_MAX;
      if (lane < ncta) {
        cv = *cluster.map_shared_rank(&cand_v[par], lane);
        ci = *cluster.map_shared_rank(&cand_i[par], lane);
      }
      warp_argmax_first_f(cv, ci);
      if (lane == 0) s_p = (ci == INT_MAX) ? kk : ci;
    }
    __syncthreads();
    const int p = s_p;
    const int own_p = p / R, loc_p = p - own_p * R;
    const int own_k = kk / R, loc_k = kk - own_k * R;
    if (tid < kLu32NB) {
      rowp[tid] = cluster.map_shared_rank(P, own_p)[loc_p * kPanelLd + tid];
    } else if (tid < 2 * kLu32NB) {
      rowk[tid - kLu32NB] = cluster.map_shared_rank(P, own_k)[loc_k * kPanelLd + tid - kLu32NB];
    }
    cluster.sync();
    const float akk = rowp[kk];
    if (akk != 0.0f && p != kk) {
      if (rank == own_k && tid < kLu32NB) P[loc_k * kPanelLd + tid] = rowp[tid];
      if (rank == own_p && tid < kLu32NB) P[loc_p * kPanelLd + tid] = rowk[tid];
    }
    if (rank == 0 && tid == 0) {
      piv[j0 + kk] = j0 + p;
      if (akk == 0.0f && *info == 0) *info = j0 + kk + 1;
    }
    __syncthreads();
    const float rcp = (akk != 0.0f) ? 1.0f / akk : 0.0f;
    for (int i = tid; i < mloc; i += blockDim.x) {
      if (r0 + i > kk) {
        float* row = P + i * kPanelLd;
        float l = row[kk];
        if (akk != 0.0f) {
          l *= rcp;
          row[kk] = l;
        }
        for (int j = kk + 1; j < nb; ++j) row[j] = fmaf(-l, rowp[j], row[j]);
      }
    }
    __syncthreads();
  }
  for (int e = tid; e < mloc * kLu32NB; e += blockDim.x) {
    const int i = e / kLu32NB, j = e % kLu32NB;
    if (j < nb) a[(int64_t)(j0 + r0 + i) * n + j0 + j] = P[i * kPanelLd + j];
  }
}

// The same panel factorisation with every panel row held in the registers of
// one thread (a CTA owns up to 512 rows, a cluster up to 16 CTAs).
//  * Rows never move: an interchange swaps the two rows' labels, and each
//    thread writes its row where its label says at the end.
//  * The columns left in a row are kept shifted: element 0 is the current
//    column, and the rank-1 update stores r[j-1] = r[j] - l prow[j].  One loop
//    body then serves all 64 columns (about 200 instructions; unrolled by
//    column the panel ran 60 times as much code once and waited for it), the
//    multipliers go to shared memory.
//  * Per column: the CTA's first max |a| by integer reductions, (key, label)
//    stored into every CTA's slots, the candidate's row laid out locally; one
//    cluster barrier; every warp picks the same winner from its own slots and
//    the winning row is read from the winner's CTA.  Slots and rows alternate
//    with the column's parity.
// Same arithmetic and pivot choice (first row of max |a|, NaN never chosen) as
// the shared-memory kernels.  Measured at m = 8192, 64 columns: 89 us (226 us with
// the columns unrolled and rows exchanged between threads).
constexpr int kRegPanelThreads = 512;
constexpr int kRegHistLd = kRegPanelThreads;
constexpr size_t kRegPanelSmem = (size_t)kLu32NB * kRegHistLd * sizeof(float);

// CLUSTER = false: a one-CTA panel (m <= 512) without cluster barriers.
template <bool CLUSTER>
__global__ void __launch_bounds__(kRegPanelThreads, 1)
panel_getf2_cluster_reg_kernel(int n, int j0, int nb, int rows_per_cta, float* __restrict__ a,
                               int32_t* __restrict__ piv, int32_t* __restrict__ info) {
  extern __shared__ __align__(16) float hist[];  // [column][thread]: multipliers
  __shared__ __align__(8) uint2 cand[2][kRegPanelThreads / 32];  // (key, label) by warp
  __shared__ __align__(8) uint2 slot[2][kPanelCluMax];           // and by CTA
  __shared__ __align__(16) float mine[2][kLu32NB];               // this CTA's candidate row
  __shared__ __align__(16) float prow[2][kLu32NB];               // the pivot row
  __shared__ int s_owner;
  cg::cluster_group cluster = cg::this_cluster();
  const int ncta = CLUSTER ? (int)cluster.num_blocks() : 1;
  const int rank = CLUSTER ? (int)cluster.block_rank() : 0;
  auto barrier = [&]() {
    if (CLUSTER) cluster.sync();
    else __syncthreads();
  };
  // shared memory of CTA `rk` of the cluster (this CTA's own without one)
  auto remote = [&](auto* ptr, int rk) { return CLUSTER ? cluster.map_shared_rank(ptr, rk) : ptr; };
  const int m = n - j0;
  const int R = rows_per_cta;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  constexpr int kWarps = kRegPanelThreads / 32;
  int gi = rank * R + tid;             // label of this thread's row
  const bool has_row = tid < R && gi < m;
  bool active = has_row;               // not yet a pivot row
  int done_at = nb;                    // columns of this row that are multipliers
  float r[kLu32NB];
#pragma unroll
  for (int j = 0; j < kLu32NB; ++j) r[j] = 0.0f;
  pdl_wait();
  pdl_trigger();  // the wide update of the step before runs beside this panel
  if (has_row) {
    const float* src = a + (int64_t)(j0 + gi) * n + j0;
    if (nb == kLu32NB) {
#pragma unroll
      for (int q = 0; q < kLu32NB / 4; ++q) {
        const float4 v = reinterpret_cast<const float4*>(src)[q];
        r[4 * q] = v.x;
        r[4 * q + 1] = v.y;
        r[4 * q + 2] = v.z;
        r[4 * q + 3] = v.w;
      }
    } else {
#pragma unroll
      for (int j = 0; j < kLu32NB; ++j) r[j] = (j < nb) ? src[j] : 0.0f;
    }
  }
  int bad = 0;
  if (CLUSTER) cluster.sync();         // every CTA runs before any remote store
#pragma unroll 1
  for (int kk = 0; kk < nb; ++kk) {
    const int par = kk & 1;
    // this CTA's first max |a| in column kk (key 0: no candidate)
    const unsigned bits = __float_as_uint(r[0]) & 0x7FFFFFFFu;
    unsigned key = (active && bits <= 0x7F800000u) ? bits + 1u : 0u;
    unsigned mk = __reduce_max_sync(0xffffffffu, key);
    unsigned ml = __reduce_min_sync(0xffffffffu, (key == mk && key != 0u) ? (unsigned)gi : ~0u);
    if (lane == 0) cand[par][warp] = make_uint2(mk, ml);
    __syncthreads();
    const uint2 w = lane < kWarps ? cand[par][lane] : make_uint2(0u, ~0u);
    mk = __reduce_max_sync(0xffffffffu, w.x);
    ml = __reduce_min_sync(0xffffffffu, w.x == mk ? w.y : ~0u);
    if (warp == 0 && lane < ncta) *remote(&slot[par][rank], lane) = make_uint2(mk, ml);
    if (active && (unsigned)gi == ml) {
#pragma unroll
      for (int q = 0; q < kLu32NB / 4; ++q)
        reinterpret_cast<float4*>(mine[par])[q] =
            make_float4(r[4 * q], r[4 * q + 1], r[4 * q + 2], r[4 * q + 3]);
    }
    barrier();                         // the one cluster barrier of this column
    const uint2 s = lane < ncta ? slot[par][lane] : make_uint2(0u, ~0u);
    mk = __reduce_max_sync(0xffffffffu, s.x);
    ml = __reduce_min_sync(0xffffffffu, s.x == mk ? s.y : ~0u);
    const bool none = mk == 0u;        // a column of NaNs: row kk stays
    const int p = none ? kk : (int)ml;
    int own = __ffs(__ballot_sync(0xffffffffu, s.x == mk && s.y == ml)) - 1;
    if (none) {                        // uniform over the cluster
      if (active && gi == kk) {
#pragma unroll
        for (int j = 0; j < kLu32NB; ++j) mine[par][j] = r[j];
        for (int c = 0; c < ncta; ++c) *remote(&s_owner, c) = rank;
      }
      barrier();
      own = s_owner;
    }
    if (warp == 0 && lane < kLu32NB / 4)
      reinterpret_cast<float4*>(prow[par])[lane] =
          reinterpret_cast<const float4*>(remote(&mine[par][0], own))[lane];
    __syncthreads();
    const float akk = prow[par][0];
    if (rank == 0 && tid == 0) {
      piv[j0 + kk] = j0 + p;
      if (akk == 0.0f && bad == 0) bad = j0 + kk + 1;
    }
    if (akk != 0.0f && p != kk) {      // the interchange: labels only
      if (gi == kk) gi = p;
      else if (gi == p) gi = kk;
    }
    if (active && gi == kk) {
      // row kk of U (written below from the pivot row; a zero pivot leaves row
      // kk where it is, and its thread writes its own row)
      active = false;
      done_at = kk;
      if (akk == 0.0f)
#pragma unroll
        for (int j = 0; j < kLu32NB; ++j)
          if (kk + j < nb) a[(int64_t)(j0 + kk) * n + j0 + kk + j] = r[j];
    }
    if (akk != 0.0f && rank == 0 && warp >= kWarps - 2) {
      const int j = (warp - (kWarps - 2)) * 32 + lane;
      if (kk + j < nb) a[(int64_t)(j0 + kk) * n + j0 + kk + j] = prow[par][j];
    }
    if (active) {
      float l = r[0];
      if (akk != 0.0f) l *= 1.0f / akk;
      hist[kk * kRegHistLd + tid] = l;
      const float4* pr = reinterpret_cast<const float4*>(prow[par]);
#pragma unroll
      for (int g = 0; g < 4; ++g) {
        if (16 * g < nb - kk) {        // the columns left, 16 at a time
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            const float4 u = pr[4 * g + q];
            const int j = 16 * g + 4 * q;
            if (j > 0) r[j - 1] = fmaf(-l, u.x, r[j]);
            r[j] = fmaf(-l, u.y, r[j + 1]);
            r[j + 1] = fmaf(-l, u.z, r[j + 2]);
            r[j + 2] = fmaf(-l, u.w, r[j + 3]);
          }
        }
      }
    }
  }
  if (rank == 0 && tid == 0 && bad != 0 && *info == 0) *info = bad;
  if (has_row) {
    float* dst = a + (int64_t)(j0 + gi) * n + j0;
    for (int c = 0; c < done_at; c += 4) {
      float v[4];
#pragma unroll
      for (int q = 0; q < 4; ++q) v[q] = (c + q < done_at) ? hist[(c + q) * kRegHistLd + tid] : 0.0f;
      if (c + 3 < done_at && (n & 3) == 0 && (j0 & 3) == 0) {
        *reinterpret_cast<float4*>(dst + c) = make_float4(v[0], v[1], v[2], v[3]);
      } else {
#pragma unroll
        for (int q = 0; q < 4; ++q)
          if (c + q < done_at) dst[c + q] = v[q];
      }
    }
  }
  if (CLUSTER) cluster.sync();  // no CTA leaves while another may still read its shared memory
}

// Cluster geometry for an m-row panel: 0 when it does not fit (or the device
// cannot co-schedule the cluster), else the CTA count (rows_per_cta set).
static int panel_cluster_size(int m, int* rows_per_cta) {
  int c = (m + kPanelCluThreads - 1) / kPanelCluThreads;
  c = c < 1 ? 1 : (c > kPanelCluMax ? kPanelCluMax : c);
  const int r = (m + c - 1) / c;
  if ((size_t)r * kPanelLd * sizeof(float) > kPanelCluSmemMax) return 0;
  *rows_per_cta = r;
  return c;
}

// Whether a cluster of c CTAs with `smem` bytes each can be co-scheduled on the
// current device (cached: the attribute and occupancy queries cost host time
// on every panel otherwise).
static bool panel_cluster_fits(int c, size_t smem) {
  static std::mutex mu;
  static std::map<std::tuple<int, int, size_t>, bool> known;
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) dev = 0;
  std::lock_guard<std::mutex> lock(mu);
  const auto key = std::make_tuple(dev, c, smem);
  auto it = known.find(key);
  if (it != known.end()) return it->second;
  bool ok = cudaFuncSetAttribute(panel_getf2_cluster_kernel,
                                 cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess &&
            ensure_dynamic_smem(reinterpret_cast<const void*>(panel_getf2_cluster_kernel),
                                (int)smem) == cudaSuccess;
  if (ok) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)c);
    cfg.blockDim = dim3(kPanelCluThreads);
    cfg.dynamicSmemBytes = smem;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = (unsigned)c;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    int nclusters = 0;
    ok = cudaOccupancyMaxActiveClusters(&nclusters, panel_getf2_cluster_kernel, &cfg) ==
             cudaSuccess &&
         nclusters >= 1;
  }
  if (!ok) cudaGetLastError();
  known[key] = ok;
  return ok;
}

// Register-resident panel when every row fits one thread of a <=16-CTA
// cluster; 0 on launch, -1 when the caller must use another kernel.
static int launch_panel_cluster_reg(int n, int j0, int nb, float* a, int32_t* piv, int32_t* info,
                                    cudaStream_t st) {
  const int m = n - j0;
  int c = (m + kRegPanelThreads - 1) / kRegPanelThreads;
  if (c < 1) c = 1;
  if (c > kPanelCluMax) return -1;
  const int r = (m + c - 1) / c;
  if (c == 1) {
    if (ensure_dynamic_smem(reinterpret_cast<const void*>(panel_getf2_cluster_reg_kernel<false>),
                            (int)kRegPanelSmem) != cudaSuccess)
      return -1;
    if (launch_pdl(panel_getf2_cluster_reg_kernel<false>, dim3(1), dim3(kRegPanelThreads),
                   kRegPanelSmem, st, 1, n, j0, nb, r, a, piv, info) == cudaSuccess)
      return 0;
  } else if (cluster_fits(reinterpret_cast<const void*>(panel_getf2_cluster_reg_kernel<true>), c,
                          kRegPanelThreads, kRegPanelSmem)) {
    if (launch_pdl(panel_getf2_cluster_reg_kernel<true>, dim3((unsigned)c), dim3(kRegPanelThreads),
                   kRegPanelSmem, st, c, n, j0, nb, r, a, piv, info) == cudaSuccess)
      return 0;
  }
  cudaGetLastError();
  return -1;
}

static int launch_panel_cluster(int n, int j0, int nb, float* a, int32_t* piv, int32_t* info,
                                cudaStream_t st) {
  if (launch_panel_cluster_reg(n, j0, nb, a, piv, info, st) == 0) return 0;
  int r = 0;
  const int c = panel_cluster_size(n - j0, &r);
  if (c == 0) return -1;
  const size_t smem = (size_t)r * kPanelLd * sizeof(float);
  if (!panel_cluster_fits(c, smem)) return -1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)c);
  cfg.blockDim = dim3(kPanelCluThreads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = (unsigned)c;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  if (cudaLaunchKernelEx(&cfg, panel_getf2_cluster_kernel, n, j0, nb, r, a, piv, info) !=
      cudaSuccess) {
    cudaGetLastError();
    return -1;
  }
  return 0;
}

__global__ void cvt_f64_to_f32_kernel(int64_t count, const double* __restrict__ src,
                                      float* __restrict__ dst) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < count;
       i += (int64_t)gridDim.x * blockDim.x)
    dst[i] = (float)src[i];
}

__global__ void zero_i32_kernel(int32_t* p, int count) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < count) p[i] = 0;
}

// getrs with an FP32 factor on FP64 vectors: x = U^{-1} L^{-1} P b, computed
// in FP32 (the preconditioner apply of GMRES-IR).  One CTA per vector.
__global__ void __launch_bounds__(256)
getrs_f32_kernel(int n, const float* __restrict__ lu, const int32_t* __restrict__ piv,
                 const double* __restrict__ b, double* __restrict__ x) {
  extern __shared__ float xs[];
  __shared__ TrsvSmem<float> tsm;
  const double* bc = b + (int64_t)blockIdx.x * n;
  double* xc = x + (int64_t)blockIdx.x * n;
  for (int i = threadIdx.x; i < n; i += blockDim.x) xs[i] = (float)bc[i];
  __syncthreads();
  if (threadIdx.x == 0)
    for (int k = 0; k < n; ++k) {
      const int p = piv[k];
      if (p != k) { const float t = xs[k]; xs[k] = xs[p]; xs[p] = t; }
    }
  __syncthreads();
  cta_trsv<float>(lu, n, n, true, false, true, xs, tsm);
  cta_trsv<float>(lu, n, n, false, false, false, xs, tsm);
  for (int i = threadIdx.x; i < n; i += blockDim.x) xc[i] = (double)xs[i];
}

}  // namespace lxgb

using namespace lxgb;

// Workspace: U12ᵀ (n×64), for 3xTF32 the hi/lo splits of L21 and U12ᵀ, for
// BF16 the BF16 copies of L21 and U12ᵀ.
extern "C" int64_t lxgb_getrf_f32_tc_workspace_size(int32_t n, int32_t precision) {
  const int64_t blk = (int64_t)(n > 0 ? n : 1) * kLu32NB * (int64_t)sizeof(float);
  const int blocks = precision == 1 ? 5 : (precision == 2 ? 4 : 1);
  return 256 + blocks * ((blk + 255) & ~(int64_t)255);
}

extern "C" int lxgb_getrf_f32_tc(int32_t n, const double* a64, float* lu, int32_t* piv,
                                 int32_t* info, int32_t precision, int32_t* err, void* work,
                                 int64_t work_bytes, void* stream) {
  LXGB_REQUIRE(precision >= 0 && precision <= 2,
               "getrf_f32_tc: precision must be 0 (TF32), 1 (3xTF32) or 2 (BF16)");
  LXGB_REQUIRE(n >= 0, "getrf_f32_tc: negative size");
  if (n == 0) return LXGB_SUCCESSFUL;
  LXGB_REQUIRE(lu && piv && info && err && work, "getrf_f32_tc: null pointer");
  LXGB_REQUIRE((n % 4) == 0, "getrf_f32_tc: n must be a multiple of 4 (16-byte TMA rows)");
  LXGB_REQUIRE((((uintptr_t)lu) & 15) == 0 && (((uintptr_t)work) & 255) == 0,
               "getrf_f32_tc: lu must be 16-byte and work 256-byte aligned");
  if (work_bytes < lxgb_getrf_f32_tc_workspace_size(n, precision)) {
    set_last_error("getrf_f32_tc: workspace too small");
    return LXGB_WORKSPACE_TOO_SMALL;
  }
  cudaStream_t st = as_stream(stream);
  if (a64) {
    const int64_t cnt = (int64_t)n * n;
    cvt_f64_to_f32_kernel<<<(unsigned)(((cnt + 255) / 256) < 8192 ? (cnt + 255) / 256 : 8192), 256,
                            0, st>>>(cnt, a64, lu);
  }
  zero_i32_kernel<<<1, 32, 0, st>>>(info, 1);
  const int64_t blk = (((int64_t)n * kLu32NB * (int64_t)sizeof(float)) + 255) & ~(int64_t)255;
  char* wb = reinterpret_cast<char*>(work) + 256;
  float* bt = reinterpret_cast<float*>(wb);
  float* ah = reinterpret_cast<float*>(wb + blk);
  float* al = reinterpret_cast<float*>(wb + 2 * blk);
  float* bh = reinterpret_cast<float*>(wb + 3 * blk);
  float* bl = reinterpret_cast<float*>(wb + 4 * blk);
  // A22 -= L21 U12 on columns [c0, c0 + cols) of the matrix, after step j0
  auto update = [&](int j0, int c0, int cols, int beside) -> int {
    const int r0 = j0 + kLu32NB, rows = n - r0;
    float* c = lu + (int64_t)r0 * n + c0;
    const int64_t at = (int64_t)(c0 - r0) * kLu32NB;  // in the operand from U12
    if (precision == 1)
      return gemm_tf32_nt_split(rows, cols, kLu32NB, ah, al, kLu32NB, bh + at, bl + at, kLu32NB, c,
                                n, -1.0f, 1.0f, err, st, beside);
    if (precision == 2)  // BF16 operands (8-bit significands), FP32 accumulation
      return gemm_bf16_nt(rows, cols, kLu32NB, ah, kLu32NB,
                          reinterpret_cast<__nv_bfloat16*>(bh) + at, kLu32NB, c, n, -1.0f, 1.0f,
                          err, st, beside);
    return gemm_tf32_nt(rows, cols, kLu32NB, lu + (int64_t)r0 * n + j0, n, bt + at, kLu32NB, c, n,
                        -1.0f, 1.0f, err, st, beside);
  };
  for (int j0 = 0; j0 < n; j0 += kLu32NB) {
    const int nb = min(kLu32NB, n - j0);
    if (launch_panel_cluster(n, j0, nb, lu, piv, info, st) != 0)
      panel_getf2_f32_kernel<<<1, kLu32PanelThreads, 0, st>>>(n, j0, nb, lu, piv, info);
    int rc = 0;
    // The columns after this panel take the step before beside the panel, which
    // leaves 136 SMs idle and is the longer of the two from n = 8192 down: 14.4
    // ms for the factor at n = 8192, 6.4 at 4096, 2.99 at 2048, against 18.9,
    // 7.0 and 3.09 with panel and update one after the other.
    if (j0 > 0 && j0 + nb < n) rc = update(j0 - kLu32NB, j0 + nb, n - j0 - nb, kBesidePanel);
    // interchanges, U12 in place and the operands of the update
    if (!rc)
      rc = lu32_block_row(precision, n, j0, nb, lu, piv, ah, al, precision == 0 ? bt : bh, bl, st);
    // the next panel's columns
    const int n2 = n - j0 - nb;
    if (!rc && n2 > 0) rc = update(j0, j0 + nb, min(kLu32NB, n2), 0);
    if (rc) return rc;
  }
  return check_launch("getrf_f32_tc");
}

extern "C" int lxgb_getrs_f32(int32_t n, int32_t nrhs, const float* lu, const int32_t* piv,
                              const double* b, double* x, void* stream) {
  LXGB_REQUIRE(n >= 0 && nrhs >= 0, "getrs_f32: negative size");
  if (n == 0 || nrhs == 0) return LXGB_SUCCESSFUL;
  LXGB_REQUIRE(lu && piv && b && x, "getrs_f32: null pointer");
  const size_t smem = (size_t)n * sizeof(float);
  LXGB_REQUIRE(smem <= 180 * 1024, "getrs_f32: n too large for the shared-memory vector");
  LXGB_CUDA_TRY(ensure_dynamic_smem(reinterpret_cast<const void*>(getrs_f32_kernel), (int)smem),
                "getrs_f32: set smem");
  getrs_f32_kernel<<<(unsigned)nrhs, 256, smem, as_stream(stream)>>>(n, lu, piv, b, x);
  return check_launch("getrs_f32");
}
