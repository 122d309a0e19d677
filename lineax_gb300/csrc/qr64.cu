// FP64 Householder QR on thread-block clusters: the factorisation of matrices
// of up to 8192 rows and the application of Q.
//
// On GB300 the FP64 pipe (2 FMA per clock and SM) bounds every phase, so the
// point is to keep many SMs on each.  Panels of 16 columns:
//   qr16_panel_kernel  — the reflectors of one panel, rows in the registers of
//                        up to 16 CTAs, one cluster exchange per column; T (16)
//   qr16_apply_kernel  — C -= V Tᵀ (Vᵀ C) on strips of columns, one cluster of
//                        CTAs per strip (rows split): C is read and written
//                        once, W = Vᵀ C is summed through distributed shared
//                        memory, nothing goes through global memory between
// Measured for 3001 x 401: 62 us a panel of 16 columns (393 us for 32 before),
// 13 us for the next panel's update, 56 us for the other columns' alone (240 us
// as three launches per 32 columns before); the factorisation 6.0 to 2.3 ms,
// Qᵀ b 3.4 to 0.1 ms.  16 columns instead of 32 halve the panel's own
// arithmetic, which only its 16 SMs share.
// The next panel's 16 columns are updated first (narrow strips, all SMs), the
// others beside the next panel: that launch depends on the panel's start only,
// reads what was finished before it and waits for the panel before it ends.
//   qr32_merge_t_kernel — the 32-column T blocks of the public factor from the
//                        pairs of 16-column ones, after the last panel.
#include <cooperative_groups.h>
#include <math.h>

#include "qr64.cuh"

namespace lxgb {

namespace cg = cooperative_groups;

constexpr int kQ16 = 16;                 // panel width
constexpr int kQTB = 32;                 // columns per public T block
constexpr int kQClu = 16;                // most CTAs per cluster
// Panel: threads that hold rows (one warp per SM sub-partition: a second would
// double the additions of the reductions), the control warp, the warp for T.
constexpr int kQRowThreads = 128;
constexpr int kQThreads = kQRowThreads + 64;
constexpr int kQGroups = kQRowThreads / 4;    // rows per register slot
constexpr int kQMaxRR = 16;              // register slots: rows per CTA / 32
// Unused dynamic shared memory that a panel CTA reserves: no CTA of the update
// running beside it shares its SM's FP64 pipe.
constexpr int kQReserve = 200 * 1024;

__device__ __forceinline__ bool is_zero(double x) {
  return (__double_as_longlong(x) << 1) == 0;  // integer test: off the FP64 pipe
}

// Reflector of a column with leading entry alpha and squared norm xn2 below it
// (LAPACK larfg): beta, tau, 1 / (alpha - beta), by a whole warp with the same
// arguments.  Where alpha² + xn2 can neither overflow nor lose digits to
// underflow, from its reciprocal root y: ||x|| = s y (corrected by one step),
// tau = 1 + |alpha| y, one division; hypot and two divisions otherwise.
__device__ __forceinline__ void larfg(double alpha, double xn2, double& beta, double& tau,
                                      double& scal) {
  if (is_zero(xn2)) {
    beta = alpha;
    tau = 0.0;
    scal = 1.0;
    return;
  }
  const unsigned ea = ((unsigned)__double2hiint(alpha) >> 20) & 0x7FFu;
  const unsigned ex = ((unsigned)__double2hiint(xn2) >> 20) & 0x7FFu;
  if (ea < 1500u && ex > 200u && ex < 1900u) {
    const double sq = fma(alpha, alpha, xn2);
    const double y = rsqrt(sq);
    double nrm = sq * y;
    nrm = fma(0.5 * y, fma(-nrm, nrm, sq), nrm);
    beta = -copysign(nrm, alpha);
    scal = 1.0 / (alpha - beta);
    tau = fma(fabs(alpha), y, 1.0);
    return;
  }
  beta = -copysign(hypot(alpha, sqrt(xn2)), alpha);
  tau = (beta - alpha) / beta;
  scal = 1.0 / (alpha - beta);
}

// Sum over the cluster of element `idx` of every CTA's shared array `p`: this
// thread takes the CTAs of parity `half` (all loads in flight at once), its
// neighbour lane the others.
__device__ __forceinline__ double cluster_sum2(const cg::cluster_group& cluster, double* p,
                                               int idx, int ncta, int half) {
  double v[kQClu / 2];
#pragma unroll
  for (int c = 0; c < kQClu / 2; ++c)
    v[c] = (2 * c + half < ncta) ? cluster.map_shared_rank(p, 2 * c + half)[idx] : 0.0;
  double s = ((v[0] + v[1]) + (v[2] + v[3])) + ((v[4] + v[5]) + (v[6] + v[7]));
  return s + __shfl_xor_sync(0xffffffffu, s, 1);
}

struct QPanelSmem {
  double part[2][kQRowThreads / 32][kQ16];  // per-warp partial dots, by column parity
  double pub[2][kQ16];                      // this CTA's dots
  double rowk[2][kQ16];                     // row k (rank 0)
  double tws[2][kQ16];                      // update coefficients below row k
  double tw[2][kQ16];                       // and in row k
  double gd[2][kQ16];                       // v_cᵀ v_k, c < k
  double sc[2][3];                          // scal, beta, tau
  int live[2];                              // tau != 0
  double T[kQ16][kQ16 + 1];
};

// Columns [j0, j0 + nb) of the factorisation, rows [j0, mm) over the cluster:
// CTA r holds rows j0 + r R .. + R; its row x lives in slot x / 32 of the four
// threads of row group x % 32, thread t of them holding columns 4 q + t.  Per
// column k: the dots of a_k below row k with all 16 columns (itself: the norm;
// earlier ones: VᵀV for T; later ones: the update) reduced over lanes, warps
// and the cluster; the control warp forms the reflector and the coefficients,
// the row threads update, another warp forms the next column of T meanwhile.
template <int RR>
__global__ void __launch_bounds__(kQThreads, 1)
qr16_panel_kernel(int64_t mm, int j0, int nb, int R, double* __restrict__ h,
                  double* __restrict__ tau, double* __restrict__ t_blk, int sub) {
  __shared__ QPanelSmem sm;
  cg::cluster_group cluster = cg::this_cluster();
  const int ncta = (int)cluster.num_blocks();
  const int rank = (int)cluster.block_rank();
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const bool holder = warp < kQRowThreads / 32;
  const bool control = warp == kQRowThreads / 32;
  const int g = (warp << 3) + (lane >> 2), t = lane & 3;
  const int64_t row0 = (int64_t)rank * R;            // first row, relative to j0
  pdl_wait();
  // everything before is finished: the update of the columns past this panel
  // may start beside it
  pdl_trigger();
  double r[RR][4];
#pragma unroll
  for (int rr = 0; rr < RR; ++rr) {
    const int x = rr * kQGroups + g;
    const bool ok = holder && x < R && j0 + row0 + x < mm;
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const int c = 4 * q + t;
      r[rr][q] = (ok && c < nb) ? h[(int64_t)(j0 + c) * mm + j0 + row0 + x] : 0.0;
    }
  }
  if (warp == kQRowThreads / 32 + 1)
    for (int e = lane; e < kQ16 * (kQ16 + 1); e += 32) (&sm.T[0][0])[e] = 0.0;
  cluster.sync();
#pragma unroll
  for (int q = 0; q < 4; ++q) {
#pragma unroll 1
    for (int tt = 0; tt < 4; ++tt) {
      const int kk = 4 * q + tt;
      if (kk >= nb) break;                           // uniform over the cluster
      const int par = kk & 1;
      double v[RR];
      if (holder) {
        double s[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll
        for (int rr = 0; rr < RR; ++rr) {
          const double a = __shfl_sync(0xffffffffu, r[rr][q], (lane & ~3) | tt);
          v[rr] = (row0 + rr * kQGroups + g > kk) ? a : 0.0;
#pragma unroll
          for (int c = 0; c < 4; ++c) s[c] = fma(v[rr], r[rr][c], s[c]);
        }
        if (rank == 0 && g == kk) {
#pragma unroll
          for (int c = 0; c < 4; ++c) sm.rowk[par][4 * c + t] = r[0][c];
        }
        // transposing butterfly over the warp's 8 rows: 4 columns -> 1 per lane
        const bool b4 = lane & 16, b3 = lane & 8;
        double k0 = b4 ? s[2] : s[0], k1 = b4 ? s[3] : s[1];
        k0 += __shfl_xor_sync(0xffffffffu, b4 ? s[0] : s[2], 16);
        k1 += __shfl_xor_sync(0xffffffffu, b4 ? s[1] : s[3], 16);
        double z = b3 ? k1 : k0;
        z += __shfl_xor_sync(0xffffffffu, b3 ? k0 : k1, 8);
        z += __shfl_xor_sync(0xffffffffu, z, 4);
        if ((lane & 4) == 0) sm.part[par][warp][4 * ((b4 ? 2 : 0) + (b3 ? 1 : 0)) + t] = z;
      }
      __syncthreads();
      const int col = lane & 15, half = lane >> 4;
      if (control) {
        static_assert(kQRowThreads / 32 == 4, "two warps' partial sums per lane");
        double p = sm.part[par][2 * half][col] + sm.part[par][2 * half + 1][col];
        p += __shfl_xor_sync(0xffffffffu, p, 16);
        if (lane < kQ16) sm.pub[par][col] = p;
      }
      cluster.sync();                                // the one cluster barrier of the column
      if (control) {
        double pv[kQClu / 2];
#pragma unroll
        for (int c = 0; c < kQClu / 2; ++c) {
          const int src = half * (kQClu / 2) + c;
          pv[c] = (src < ncta) ? cluster.map_shared_rank(&sm.pub[par][0], src)[col] : 0.0;
        }
        const double rk = cluster.map_shared_rank(&sm.rowk[par][0], 0)[col];
        double d = ((pv[0] + pv[1]) + (pv[2] + pv[3])) + ((pv[4] + pv[5]) + (pv[6] + pv[7]));
        d += __shfl_xor_sync(0xffffffffu, d, 16);
        const double xn2 = __shfl_sync(0xffffffffu, d, kk);
        const double alpha = __shfl_sync(0xffffffffu, rk, kk);
        double beta, scal, tk;
        larfg(alpha, xn2, beta, tk, scal);
        // v_kᵀ a_c = a_c[k] + scal d_c (v_k[k] = 1); for c < k the same sum is v_cᵀ v_k
        d = fma(scal, d, rk);
        const double tw = tk * d;
        if (lane < kQ16) {
          sm.tw[par][col] = tw;
          sm.tws[par][col] = tw * scal;
          sm.gd[par][col] = d;
        }
        if (lane == 0) {
          sm.sc[par][0] = scal;
          sm.sc[par][1] = beta;
          sm.sc[par][2] = tk;
          sm.live[par] = !is_zero(tk);
          if (rank == 0) tau[j0 + kk] = tk;
        }
      }
      __syncthreads();
      if (warp == kQRowThreads / 32 + 1) {
        // T[0:k, k] = -tau T[0:k, 0:k] (V[:, 0:k]ᵀ v_k), T[k][k] = tau
        const double tk = sm.sc[par][2];
        double acc = 0.0;
        for (int p = 0; p < kk; ++p)
          if (lane < kk) acc = fma(sm.T[lane][p], sm.gd[par][p], acc);
        if (lane < kk) sm.T[lane][kk] = -tk * acc;
        if (lane == kk) sm.T[kk][kk] = tk;
        __syncwarp();
      } else if (holder && sm.live[par]) {
        const double scal = sm.sc[par][0];
        const bool rowk = rank == 0 && g == kk;
#pragma unroll
        for (int c = q; c < 4; ++c) {
          if (c > q || t > tt) {
            const double w = sm.tws[par][4 * c + t];
            // (rows up to kk are in the first slot; their v is 0, w may be infinite or NaN)
#pragma unroll
            for (int rr = 0; rr < RR; ++rr)
              if (rr > 0 || row0 + g > kk) r[rr][c] = fma(-w, v[rr], r[rr][c]);
            if (rowk) r[0][c] -= sm.tw[par][4 * c + t];
          }
        }
        if (t == tt) {
#pragma unroll
          for (int rr = 0; rr < RR; ++rr)
            if (row0 + rr * kQGroups + g > kk) r[rr][q] = v[rr] * scal;
          if (rowk) r[0][q] = sm.sc[par][1];
        }
      }
    }
  }
#pragma unroll
  for (int rr = 0; rr < RR; ++rr) {
    const int x = rr * kQGroups + g;
    const bool ok = holder && x < R && j0 + row0 + x < mm;
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const int c = 4 * q + t;
      if (ok && c < nb) h[(int64_t)(j0 + c) * mm + j0 + row0 + x] = r[rr][q];
    }
  }
  __syncthreads();
  if (rank == 0) {
    // the panel's T on the diagonal of its 32-column block; the first panel of
    // a block clears the rest
    for (int e = tid; e < kQTB * kQTB; e += kQThreads) {
      const int i = e / kQTB, j = e % kQTB;
      const bool in = (i / kQ16 == sub) && (j / kQ16 == sub);
      if (in) t_blk[e] = sm.T[i % kQ16][j % kQ16];
      else if (sub == 0) t_blk[e] = 0.0;
    }
  }
  cluster.sync();  // no CTA leaves while another may still read its shared memory
}

// C -= V Tᵀ (Vᵀ C) for columns [c_lo, c_hi) of the trailing matrix and the panel
// at j0: strip blockIdx.x / ncta of S columns, rows split over the cluster.
// V (16 wide) and the strip are staged in shared memory, rows outermost.
// BESIDE: this launch runs beside the next panel (see above).
constexpr int kQaThreads = 256;
constexpr int kQaLd = 18;  // doubles per staged row of V: 16-byte aligned, spreads the banks

template <int S, bool BESIDE>
__global__ void __launch_bounds__(kQaThreads, 3)
qr16_apply_kernel(int64_t mm, int j0, int nb, int R, int c_lo, int c_hi, double* h,
                  const double* t_blk, int sub) {
  extern __shared__ __align__(16) double qa_dyn[];
  constexpr int O = kQ16 * S;               // outputs of W
  constexpr int kWarps = kQaThreads / 32;
  static_assert(kWarps == 8 && 2 * O <= kQaThreads, "two threads per output of W");
  __shared__ double part[kWarps][O];
  __shared__ double pub[O], W[O], W2[O];
  __shared__ double T[kQ16][kQ16 + 1];
  cg::cluster_group cluster = cg::this_cluster();
  const int ncta = (int)cluster.num_blocks();
  const int rank = (int)cluster.block_rank();
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int c0 = c_lo + (int)(blockIdx.x / ncta) * S;
  const int64_t lo = j0 + (int64_t)rank * R;
  const int rows = (int)max((int64_t)0, min((int64_t)R, mm - lo));
  double* V = qa_dyn;                       // rows × kQaLd
  double* C = qa_dyn + (int64_t)R * kQaLd;  // S × R
  if (!BESIDE) pdl_wait();
  auto ld = [&](const double* p) { return BESIDE ? __ldcg(p) : *p; };
  // all loads of a row are in flight before the first is stored
  static_assert(kQaThreads == kQ16 * kQ16, "one entry of T per thread");
  const double te =
      ld(t_blk + (sub * kQ16 + tid / kQ16) * kQTB + sub * kQ16 + tid % kQ16);
  for (int x = tid; x < rows; x += kQaThreads) {
    const int64_t i = lo + x;
    double v[kQ16], cv[S];
#pragma unroll
    for (int p = 0; p < kQ16; ++p)
      v[p] = (p < nb && i > j0 + p) ? ld(h + (int64_t)(j0 + p) * mm + i)
                                    : ((p < nb && i == j0 + p) ? 1.0 : 0.0);
#pragma unroll
    for (int s = 0; s < S; ++s)
      cv[s] = (c0 + s < c_hi) ? ld(h + (int64_t)(c0 + s) * mm + i) : 0.0;
#pragma unroll
    for (int p = 0; p < kQ16; p += 2)
      *reinterpret_cast<double2*>(V + x * kQaLd + p) = make_double2(v[p], v[p + 1]);
#pragma unroll
    for (int s = 0; s < S; ++s) C[s * R + x] = cv[s];
  }
  T[tid / kQ16][tid % kQ16] = te;
  __syncthreads();
  // W = Vᵀ C over this CTA's rows: warp w the rows w mod 8, a lane O / 32 outputs
  if (S == 8) {
    const int pl = (lane >> 3) * 4, sl = lane & 7;
    double acc[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll 2
    for (int x = warp; x < rows; x += kWarps) {
      const double c = C[sl * R + x];
      const double2 v0 = *reinterpret_cast<const double2*>(V + x * kQaLd + pl);
      const double2 v1 = *reinterpret_cast<const double2*>(V + x * kQaLd + pl + 2);
      acc[0] = fma(v0.x, c, acc[0]);
      acc[1] = fma(v0.y, c, acc[1]);
      acc[2] = fma(v1.x, c, acc[2]);
      acc[3] = fma(v1.y, c, acc[3]);
    }
#pragma unroll
    for (int k = 0; k < 4; ++k) part[warp][(pl + k) * S + sl] = acc[k];
  } else {
    const int pl = lane / S, sl = lane % S;         // S == 2: one output per lane
    double acc[2] = {0.0, 0.0};
    int x = warp;
    for (; x + kWarps < rows; x += 2 * kWarps) {
      acc[0] = fma(V[x * kQaLd + pl], C[sl * R + x], acc[0]);
      acc[1] = fma(V[(x + kWarps) * kQaLd + pl], C[sl * R + x + kWarps], acc[1]);
    }
    if (x < rows) acc[0] = fma(V[x * kQaLd + pl], C[sl * R + x], acc[0]);
    part[warp][pl * S + sl] = acc[0] + acc[1];
  }
  __syncthreads();
  const int o2 = tid >> 1, half = tid & 1;          // two threads per output
  if (tid < 2 * O) {
    double s = (part[half][o2] + part[half + 2][o2]) + (part[half + 4][o2] + part[half + 6][o2]);
    s += __shfl_xor_sync(0xffffffffu, s, 1);
    if (half == 0) pub[o2] = s;
  }
  cluster.sync();
  if (tid < 2 * O) {
    const double s = cluster_sum2(cluster, pub, o2, ncta, half);
    if (half == 0) W[o2] = s;
  }
  __syncthreads();
  if (tid < O) {
    const int p = tid / S, s = tid % S;
    double acc[2] = {0.0, 0.0};                      // row p of Tᵀ: T[q][p], q <= p
#pragma unroll
    for (int q = 0; q < kQ16; ++q)
      if (q <= p) acc[q & 1] = fma(T[q][p], W[q * S + s], acc[q & 1]);
    W2[tid] = acc[0] + acc[1];
  }
  __syncthreads();
  if (!BESIDE) pdl_trigger();
  for (int e = tid; e < rows * S; e += kQaThreads) {
    const int s = e / rows, x = e - s * rows;
    if (c0 + s >= c_hi) break;
    double acc[2] = {C[s * R + x], 0.0};
    const double2* v = reinterpret_cast<const double2*>(V + x * kQaLd);
#pragma unroll
    for (int p = 0; p < kQ16 / 2; ++p) {
      const double2 vv = v[p];
      acc[0] = fma(-W2[(2 * p) * S + s], vv.x, acc[0]);
      acc[1] = fma(-W2[(2 * p + 1) * S + s], vv.y, acc[1]);
    }
    h[(int64_t)(c0 + s) * mm + lo + x] = acc[0] + acc[1];
  }
  cluster.sync();  // no CTA leaves while another may still read its shared memory
  if (BESIDE) pdl_wait();
}

// T of a 32-column block from its two 16-column ones: T_AB = -T_A (V_Aᵀ V_B) T_B.
// One cluster per block, rows split; thread (p, q) sums its product over the
// rows staged 64 at a time.
__global__ void __launch_bounds__(256)
qr32_merge_t_kernel(int64_t mm, int nn, const double* __restrict__ h, double* __restrict__ t) {
  __shared__ double V[64][kQTB + 1];
  __shared__ double G[kQ16][kQ16 + 1], X[kQ16][kQ16 + 1];
  cg::cluster_group cluster = cg::this_cluster();
  const int ncta = (int)cluster.num_blocks();
  const int rank = (int)cluster.block_rank();
  const int blk = (int)(blockIdx.x / ncta);
  const int j0 = blk * kQTB;
  const int nb = min(kQTB, nn - j0);
  double* T = t + (int64_t)blk * kQTB * kQTB;
  const int tid = threadIdx.x, p = tid / kQ16, q = tid % kQ16;
  pdl_wait();
  const int64_t first = j0 + kQ16;           // rows above hold zeros of V_B
  const int64_t span = mm - first;
  const int64_t R = (span + ncta - 1) / ncta;
  const int64_t lo = first + rank * R, hi = min(mm, lo + R);
  double acc[2] = {0.0, 0.0};
  for (int64_t i0 = lo; i0 < hi; i0 += 64) {
    double v[64 * kQTB / 256];
#pragma unroll
    for (int u = 0; u < 64 * kQTB / 256; ++u) {
      const int e = tid + 256 * u, c = e / 64;
      const int64_t i = i0 + e % 64;
      v[u] = (c < nb && i < hi && i > j0 + c) ? h[(int64_t)(j0 + c) * mm + i]
                                              : ((c < nb && i == j0 + c) ? 1.0 : 0.0);
    }
#pragma unroll
    for (int u = 0; u < 64 * kQTB / 256; ++u) V[(tid + 256 * u) % 64][(tid + 256 * u) / 64] = v[u];
    __syncthreads();
#pragma unroll 8
    for (int x = 0; x < 64; x += 2) {
      acc[0] = fma(V[x][p], V[x][kQ16 + q], acc[0]);
      acc[1] = fma(V[x + 1][p], V[x + 1][kQ16 + q], acc[1]);
    }
    __syncthreads();
  }
  G[p][q] = acc[0] + acc[1];
  cluster.sync();
  if (rank == 0) {
    double v[kQClu];
#pragma unroll
    for (int c = 0; c < kQClu; ++c)
      v[c] = (c < ncta) ? cluster.map_shared_rank(&G[0][0], c)[p * (kQ16 + 1) + q] : 0.0;
#pragma unroll
    for (int o = 1; o < kQClu; o *= 2)
#pragma unroll
      for (int c = 0; c + o < kQClu; c += 2 * o) v[c] += v[c + o];
    X[p][q] = v[0];
    __syncthreads();
    double y = 0.0;                            // (G T_B)[p][q]
    for (int k = 0; k <= q; ++k) y = fma(X[p][k], T[(kQ16 + k) * kQTB + kQ16 + q], y);
    __syncthreads();
    X[p][q] = y;
    __syncthreads();
    double z = 0.0;
    for (int k = p; k < kQ16; ++k) z = fma(T[p * kQTB + k], X[k][q], z);
    T[p * kQTB + kQ16 + q] = -z;
  }
  cluster.sync();
}

// op(Q) c for one vector per cluster: the CTA's rows of c stay in shared memory
// over all panels.  Per 32-column panel: warp w forms the dots of reflectors
// 4 w .. 4 w + 3 with the CTA's rows, the cluster sums them, every CTA applies
// T (or Tᵀ) and subtracts V w', the eight warps' shares meeting in shared
// memory.  One launch instead of two per panel.
constexpr int kOmThreads = 256;
constexpr int kOmSlots = 6;          // rows per lane held in registers
constexpr int kOmMaxRows = 2048;     // rows per CTA: 9 doubles of shared memory each
constexpr int kOmManyRows = 1024;    // of many vectors: two CTAs per SM

__global__ void __launch_bounds__(kOmThreads)
ormqr_cluster_kernel(int64_t mm, int nn, int R, const double* __restrict__ h,
                     const double* __restrict__ t, int trans, double* __restrict__ cvec) {
  extern __shared__ __align__(16) double om_dyn[];
  __shared__ double dots[2][kQTB], w[kQTB], w2[kQTB];
  cg::cluster_group cluster = cg::this_cluster();
  const int ncta = (int)cluster.num_blocks();
  const int rank = (int)cluster.block_rank();
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  double* c = om_dyn;                 // R
  double* part = om_dyn + R;          // 8 × R
  double* g = cvec + (int64_t)blockIdx.y * mm;
  const int64_t lo = (int64_t)rank * R;
  const int rows = (int)max((int64_t)0, min((int64_t)R, mm - lo));
  pdl_wait();
  for (int x = tid; x < rows; x += kOmThreads) c[x] = g[lo + x];
  __syncthreads();
  const int npan = (nn + kQTB - 1) / kQTB;
  for (int s = 0; s < npan; ++s) {
    const int pidx = trans ? s : npan - 1 - s;
    const int j0 = pidx * kQTB;
    const int par = s & 1;
    const int first = (int)max((int64_t)0, j0 - lo);  // rows above hold zeros of V
    auto vel = [&](int p, int64_t i) {
      return (j0 + p >= nn || i < j0 + p) ? 0.0
                                          : (i == j0 + p ? 1.0 : h[(int64_t)(j0 + p) * mm + i]);
    };
    // this thread's entries of op(T): output tid / 8, inputs 4 (tid % 8) ..
    const int op = tid >> 3, oq = (tid & 7) * 4;
    double tv[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const double* T = t + (int64_t)pidx * kQTB * kQTB;
      tv[k] = trans ? T[(oq + k) * kQTB + op] : T[op * kQTB + oq + k];
    }
    // V in registers, kOmSlots rows per lane at a time; a slice of at most 32
    // kOmSlots rows is loaded once for both passes
    double v[kOmSlots][4];
    auto load = [&](int x0) {
#pragma unroll
      for (int u = 0; u < kOmSlots; ++u) {
        const int x = x0 + 32 * u + lane;
#pragma unroll
        for (int k = 0; k < 4; ++k) v[u][k] = (x < rows) ? vel(4 * warp + k, lo + x) : 0.0;
      }
    };
    double a[4] = {0.0, 0.0, 0.0, 0.0};
    const bool once = rows - first <= 32 * kOmSlots;
    for (int x0 = first; x0 < rows; x0 += 32 * kOmSlots) {
      load(x0);
#pragma unroll
      for (int u = 0; u < kOmSlots; ++u) {
        const int x = x0 + 32 * u + lane;
        const double cx = (x < rows) ? c[x] : 0.0;
#pragma unroll
        for (int k = 0; k < 4; ++k) a[k] = fma(v[u][k], cx, a[k]);
      }
    }
    {
      // transposing butterfly: 4 dots over 32 lanes
      const bool b4 = lane & 16, b3 = lane & 8;
      double k0 = b4 ? a[2] : a[0], k1 = b4 ? a[3] : a[1];
      k0 += __shfl_xor_sync(0xffffffffu, b4 ? a[0] : a[2], 16);
      k1 += __shfl_xor_sync(0xffffffffu, b4 ? a[1] : a[3], 16);
      double z = b3 ? k1 : k0;
      z += __shfl_xor_sync(0xffffffffu, b3 ? k0 : k1, 8);
#pragma unroll
      for (int o = 4; o > 0; o >>= 1) z += __shfl_xor_sync(0xffffffffu, z, o);
      if ((lane & 7) == 0) dots[par][4 * warp + (b4 ? 2 : 0) + (b3 ? 1 : 0)] = z;
    }
    cluster.sync();
    if (tid < 2 * kQTB) {
      const double z = cluster_sum2(cluster, &dots[par][0], tid >> 1, ncta, tid & 1);
      if ((tid & 1) == 0) w[tid >> 1] = z;
    }
    __syncthreads();
    {
      double z = 0.0;
#pragma unroll
      for (int k = 0; k < 4; ++k) z = fma(tv[k], w[oq + k], z);
#pragma unroll
      for (int o = 4; o > 0; o >>= 1) z += __shfl_xor_sync(0xffffffffu, z, o);
      if ((tid & 7) == 0) w2[op] = z;
    }
    __syncthreads();
    for (int x0 = first; x0 < rows; x0 += 32 * kOmSlots) {
      if (!once) load(x0);
#pragma unroll
      for (int u = 0; u < kOmSlots; ++u) {
        const int x = x0 + 32 * u + lane;
        double y = 0.0;
#pragma unroll
        for (int k = 0; k < 4; ++k) y = fma(v[u][k], w2[4 * warp + k], y);
        if (x < rows) part[warp * R + x] = y;
      }
    }
    __syncthreads();
    for (int x = first + tid; x < rows; x += kOmThreads) {
      double y = c[x];
#pragma unroll
      for (int k = 0; k < kOmThreads / 32; ++k) y -= part[k * R + x];
      c[x] = y;
    }
    __syncthreads();
  }
  for (int x = tid; x < rows; x += kOmThreads) g[lo + x] = c[x];
  cluster.sync();  // no CTA leaves while another may still read its dots
}

// --- launches -----------------------------------------------------------------

template <int RR>
static cudaError_t panel_launch(int c, int R, int64_t m, int j0, int nb, double* h, double* tau,
                                double* t_blk, int sub, cudaStream_t st) {
  return launch_pdl(qr16_panel_kernel<RR>, dim3((unsigned)c), dim3(kQThreads), kQReserve, st, c, m,
                    j0, nb, R, h, tau, t_blk, sub);
}

// CTAs and rows per CTA of a panel with `rows` rows: about 64 rows each or
// more, never below 16 (row k of the panel always belongs to CTA 0).
static void panel_geometry(int64_t rows, int* c, int* R) {
  int64_t n = (rows + 63) / 64;
  if (n > kQClu) n = kQClu;
  *R = (int)((rows + n - 1) / n);
  if (*R < kQ16) *R = kQ16;
  *c = (int)((rows + *R - 1) / *R);
}

static const void* panel_fn(int rr) {
  switch (rr) {
    case 1: return reinterpret_cast<const void*>(qr16_panel_kernel<1>);
    case 2: return reinterpret_cast<const void*>(qr16_panel_kernel<2>);
    case 3: return reinterpret_cast<const void*>(qr16_panel_kernel<3>);
    case 4: return reinterpret_cast<const void*>(qr16_panel_kernel<4>);
    case 6: return reinterpret_cast<const void*>(qr16_panel_kernel<6>);
    case 8: return reinterpret_cast<const void*>(qr16_panel_kernel<8>);
    case 12: return reinterpret_cast<const void*>(qr16_panel_kernel<12>);
    default: return reinterpret_cast<const void*>(qr16_panel_kernel<16>);
  }
}

static int panel_slots(int R) {
  const int rr = (R + kQGroups - 1) / kQGroups;
  return rr <= 4 ? rr : (rr <= 6 ? 6 : (rr <= 8 ? 8 : (rr <= 12 ? 12 : 16)));
}

// CTAs per strip of the update: about `aim` rows each, at most 16 CTAs.
static void apply_geometry(int64_t rows, int aim, int* c, int* R) {
  int64_t n = (rows + aim - 1) / aim;
  if (n > kQClu) n = kQClu;
  if (n < 1) n = 1;
  *R = (int)((rows + n - 1) / n);
  *c = (int)((rows + *R - 1) / *R);
}

template <int S>
static size_t apply_smem(int R) {
  return (size_t)R * (kQaLd + S) * sizeof(double);
}

// Rows per CTA aimed at: 64 for the next panel's strips (2 columns each; their
// time is on the critical path, so as many CTAs as a cluster may have; 32 and 128
// measure the same within 1 %), 320 for the others (8 columns each).  Small strips make
// clusters of 16, which find fewer places beside the panel's; large ones hold few CTAs
// per SM.  us for the factor with 188, 320, 500 and 700 rows: 1000 x 1000 4164, 3947,
// 3817, 3811; 2000 x 500 2583, 2539, 2365, 2547; 3001 x 401 2568, 2398, 2266, 2485;
// 5000 x 1000 15860, 16530, 14520, 17760; 8192 x 2000 87440, 87450, 91480, 106700.
// 320 is never far off; 500 is better below 8192 rows.
constexpr int kQNextRows = 64, kQWideRows = 320;

int geqrf64_cluster(int64_t m, int n, double* h, double* tau, double* t, cudaStream_t st) {
  // 16 register slots of 32 rows in each of 16 CTAs; the update's staged rows
  // then fit its 8 CTAs' shared memory as well
  if (m > (int64_t)kQClu * kQGroups * kQMaxRR || n < 2) return -1;
  // every shape of the sweep has to be schedulable before the first launch
  for (int j0 = 0; j0 < n; j0 += kQ16) {
    int c, R;
    panel_geometry(m - j0, &c, &R);
    if (!cluster_fits(panel_fn(panel_slots(R)), c, kQThreads, kQReserve)) return -1;
    if (n - j0 <= kQ16) break;
    if (!cluster_fits(reinterpret_cast<const void*>(qr32_merge_t_kernel), kQClu, 256, 0)) return -1;
    apply_geometry(m - j0, kQNextRows, &c, &R);
    if (!cluster_fits(reinterpret_cast<const void*>(qr16_apply_kernel<2, false>), c, kQaThreads,
                      apply_smem<2>(R)))
      return -1;
    apply_geometry(m - j0, kQWideRows, &c, &R);
    if (!cluster_fits(reinterpret_cast<const void*>(qr16_apply_kernel<8, true>), c, kQaThreads,
                      apply_smem<8>(R)))
      return -1;
  }
  auto tblk = [&](int j0) { return t + (int64_t)(j0 / kQTB) * kQTB * kQTB; };
  auto panel = [&](int j0) -> cudaError_t {
    const int nb = n - j0 < kQ16 ? n - j0 : kQ16;
    int c, R;
    panel_geometry(m - j0, &c, &R);
    const int sub = (j0 / kQ16) & 1;
    switch (panel_slots(R)) {
      case 1: return panel_launch<1>(c, R, m, j0, nb, h, tau, tblk(j0), sub, st);
      case 2: return panel_launch<2>(c, R, m, j0, nb, h, tau, tblk(j0), sub, st);
      case 3: return panel_launch<3>(c, R, m, j0, nb, h, tau, tblk(j0), sub, st);
      case 4: return panel_launch<4>(c, R, m, j0, nb, h, tau, tblk(j0), sub, st);
      case 6: return panel_launch<6>(c, R, m, j0, nb, h, tau, tblk(j0), sub, st);
      case 8: return panel_launch<8>(c, R, m, j0, nb, h, tau, tblk(j0), sub, st);
      case 12: return panel_launch<12>(c, R, m, j0, nb, h, tau, tblk(j0), sub, st);
      default: return panel_launch<16>(c, R, m, j0, nb, h, tau, tblk(j0), sub, st);
    }
  };
  LXGB_CUDA_TRY(panel(0), "geqrf: panel launch");
  for (int j0 = 0; n - j0 > kQ16; j0 += kQ16) {
    const int s = j0 + kQ16;                         // first trailing column
    const int next = n - s < kQ16 ? n - s : kQ16;
    const int sub = (j0 / kQ16) & 1;
    int c, R;
    apply_geometry(m - j0, kQNextRows, &c, &R);
    LXGB_CUDA_TRY(launch_pdl(qr16_apply_kernel<2, false>, dim3((unsigned)((next + 1) / 2 * c)),
                             dim3(kQaThreads), apply_smem<2>(R), st, c, m, j0, kQ16, R, s, s + next,
                             h, tblk(j0), sub),
                  "geqrf: next panel update launch");
    LXGB_CUDA_TRY(panel(s), "geqrf: panel launch");
    const int rest = n - s - next;
    if (rest > 0) {
      apply_geometry(m - j0, kQWideRows, &c, &R);
      LXGB_CUDA_TRY(launch_pdl(qr16_apply_kernel<8, true>, dim3((unsigned)((rest + 7) / 8 * c)),
                               dim3(kQaThreads), apply_smem<8>(R), st, c, m, j0, kQ16, R, s + next,
                               n, h, tblk(j0), sub),
                    "geqrf: trailing update launch");
    }
  }
  // the 32-column T blocks that hold two panels
  const int pairs = n / kQTB + (n % kQTB > kQ16 ? 1 : 0);
  if (pairs > 0) {
    int c = (int)((m + 127) / 128);
    if (c > kQClu) c = kQClu;
    LXGB_CUDA_TRY(launch_pdl(qr32_merge_t_kernel, dim3((unsigned)(pairs * c)), dim3(256), 0, st, c,
                             m, n, h, t),
                  "geqrf: T merge launch");
  }
  return check_launch("geqrf");
}

int ormqr64_cluster(int64_t m, int n, const double* h, const double* t, int nrhs, double* c,
                    int trans, cudaStream_t st) {
  int64_t ctas = (m + 127) / 128;
  if (ctas > kQClu) ctas = kQClu;
  // One vector wants many CTAs.  With more of them than eight per SM what counts is the
  // work between a panel's two cluster barriers, so the rows go to fewer CTAs, up to
  // kOmManyRows each.  us for 500 vectors with 16, 8, 4, 2 and 1: 2000 x 2000 20250,
  // 14937, 10958, 8835, 8524 (two launches per panel: 11965), 8192 x 64 2028, 1499, 1848
  // (2334).
  while (ctas > 1 && nrhs * ctas > 8LL * sm_count() &&
         (m + ctas / 2 - 1) / (ctas / 2) <= kOmManyRows)
    ctas /= 2;
  const int64_t R = (m + ctas - 1) / ctas;
  if (R > kOmMaxRows) return -1;
  const size_t smem = (size_t)R * (1 + kOmThreads / 32) * sizeof(double);
  const void* fn = reinterpret_cast<const void*>(ormqr_cluster_kernel);
  if (!cluster_fits(fn, (int)ctas, kOmThreads, smem)) return -1;
  LXGB_CUDA_TRY(launch_pdl(ormqr_cluster_kernel, dim3((unsigned)ctas, (unsigned)nrhs),
                           dim3(kOmThreads), smem, st, (int)ctas, m, n, (int)R, h, t, trans, c),
                "ormqr: launch");
  return check_launch("ormqr");
}

}  // namespace lxgb
