// Multi-CTA FP64 triangular solve, right-looking by blocks of 64 unknowns.
//
// Unknowns are numbered in solve order (u = 0 is solved first: row u of a
// lower op(T), row n - 1 - u of an upper one), so every case is a forward
// substitution with the matrix op(u, v) = op(T)[row(u)][row(v)], v <= u.
// Launch b of the chain
//   * CTA 0: subtracts block b-1's contribution from block b and solves it;
//   * CTAs 1..: subtract block b-1's contribution from the rows after block b,
//     64 rows each.
// So each block costs one launch; matrix entries are loaded into registers
// before the kernel waits for the launch before it (they do not depend on it).
//
// What bounds it: the chain of CTA 0.  A 64-unknown step takes about 8 us:
// two 32-step substitutions by one warp (a shuffle and a dependent FP64 FMA
// per step), the 64x64 update (2 FP64 FMA per clock and SM: 1 us) and the
// hand-over between launches.  Four lanes share a row in the updates: 16 FMAs
// and two shuffle additions per lane, against 2 FMAs and five additions with
// a warp per row.  Measured (five vectors, us): n = 128 23, n = 1000 135, n =
// 2003 282; one CTA per vector with a division per unknown took 68 and 452 at
// n = 128 and 767, and a diagonal and an update launch per block 549 and 1104
// at n = 1000 and 2003.
// Few vectors of up to 2048 unknowns: trisolve_cluster_kernel below; many of up to
// 4096: trisolve_many_kernel.
#include <cooperative_groups.h>

#include "trisolve.cuh"

namespace lxgb {

namespace cg = cooperative_groups;

constexpr int kTsThreads = 256;

struct TsView {
  const double* t;
  int64_t ldt;
  int n;
  bool fwd, trans;
  __device__ __forceinline__ int64_t row(int u) const { return fwd ? u : n - 1 - u; }
  __device__ __forceinline__ double op(int u, int v) const {
    const int64_t i = row(u), j = row(v);
    return trans ? t[j * ldt + i] : t[i * ldt + j];
  }
  __device__ __forceinline__ const double* at(int u, int v) const {
    const int64_t i = row(u), j = row(v);
    return t + (trans ? j * ldt + i : i * ldt + j);
  }
};

// Whether x is zero or of moderate size (2^-500 < |x| < 2^500), by its exponent.
__device__ __forceinline__ bool ts_moderate(double x, bool zero_ok) {
  const unsigned hi = (unsigned)__double2hiint(x) & 0x7FFFFFFFu;
  const unsigned e = hi >> 20;
  if (zero_ok && hi == 0u && __double2loint(x) == 0) return true;
  return e > 523u && e < 1523u;
}

// v / dd from rinv, the rounded reciprocal of a moderate dd: the product and one step
// on its exact residual, which rounds as the quotient does (Markstein, IBM J. Res.
// Dev. 34, 1990; 3e8 random pairs on the CPU: no difference).  Two FMAs more in the
// chain than the product alone; a division took about 0.3 us a block (LU solve at
// n = 1000 2.29 ms, with the product 2.26).
__device__ __forceinline__ double ts_quotient(double v, double dd, double rinv) {
  if (!ts_moderate(v, true)) return v / dd;
  const double q = v * rinv;
  const double x = fma(fma(-q, dd, v), rinv, q);
  return ts_moderate(v, false) ? x : q;            // a zero keeps its sign
}

// One warp solves a 32-unknown block: lane l holds v = b_l and d[t] = op(l, t)
// (0 for t >= l, or past the block's end), dd = op(l, l) (1 for unit
// diagonals and past the end), and for moderate entries rinv = 1 / dd.
//  * kTsScaled: d[t] was multiplied by 1/op(t, t), so a step is v_l -= d[t] v_t on
//    unscaled v: a shuffle and an FMA, and the quotients x_l = v_l / op(l, l) of all
//    lanes come at the end.  Forward errors against 128 bits (n = 32 to 300, mean over
//    40 systems of three kinds): those of a division per step, within 3 % either way;
//    with the bare product by the reciprocal at the end up to 10 % above.
//  * kTsQuotient (one block of 64): x_t is rounded before it is used, as with a division
//    per step.  Up to n = 16 the scaled form's backward errors are 10 to 20 %
//    larger, from n = 33 on the same.
//  * kTsDivide (entries whose scaling could overflow or underflow, zeros and non-finite
//    values on the diagonal): every unknown is divided in turn.
// Lanes already solved take no part in a step, so a non-finite unknown leaves them alone.
enum TsForm { kTsScaled, kTsQuotient, kTsDivide };

__device__ __forceinline__ TsForm ts_form(int n, bool moderate) {
  return !moderate ? kTsDivide : (n <= kTsNB ? kTsQuotient : kTsScaled);
}

// V vectors side by side; d in registers or, D[t][l], in shared memory; m: the block's
// unknowns, uniform.
__device__ __forceinline__ double ts_coef(const double (&d)[32], int t, int) { return d[t]; }
__device__ __forceinline__ double ts_coef(const double (&d)[32][33], int t, int lane) {
  return d[t][lane];
}

template <int V, typename Coef>
__device__ __forceinline__ void ts_solve32(double (&v)[V], const Coef& d, int m, double dd,
                                           double rinv, bool unit, TsForm form) {
  constexpr bool kRegs = sizeof(Coef) == 32 * sizeof(double);  // all steps: d holds zeros
  const int lane = threadIdx.x & 31;
  if (form == kTsScaled) {
#pragma unroll
    for (int t = 0; t < 31; ++t) {
      if (!kRegs && t + 1 >= m) break;
      double vt[V];
#pragma unroll
      for (int q = 0; q < V; ++q) vt[q] = __shfl_sync(0xffffffffu, v[q], t);
#pragma unroll
      for (int q = 0; q < V; ++q)
        if (lane > t) v[q] = fma(-ts_coef(d, t, lane), vt[q], v[q]);
    }
#pragma unroll
    for (int q = 0; q < V; ++q)
      if (!unit) v[q] = ts_quotient(v[q], dd, rinv);
    return;
  }
  const bool quick = form == kTsQuotient;
#pragma unroll
  for (int t = 0; t < 32; ++t) {
    if (t >= m) break;
#pragma unroll
    for (int q = 0; q < V; ++q) {
      double xt = 0.0;
      if (lane == t) xt = quick ? ts_quotient(v[q], dd, rinv) : v[q] / dd;
      xt = __shfl_sync(0xffffffffu, xt, t);
      if (lane == t) v[q] = xt;
      if (lane > t) v[q] = fma(-ts_coef(d, t, lane), xt, v[q]);
    }
  }
}

__device__ __forceinline__ double ts_solve32(double v, const double (&d)[32], int m, double dd,
                                             double rinv, bool unit, TsForm form) {
  double w[1] = {v};
  ts_solve32(w, d, m, dd, rinv, unit, form);
  return w[0];
}

__global__ void __launch_bounds__(kTsThreads)
trisolve_step_kernel(int n, const double* __restrict__ t, int64_t ldt, int64_t stride_t,
                     int fwd, int trans, int unit, int b, double* __restrict__ x,
                     int64_t stride_x) {
  __shared__ double xp[kTsNB], xc[kTsNB];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const TsView T{t + (int64_t)blockIdx.z * stride_t, ldt, n, fwd != 0, trans != 0};
  double* xv = x + (int64_t)blockIdx.z * stride_x + (int64_t)blockIdx.y * n;
  const int u0 = b * kTsNB;
  const int p0 = u0 - kTsNB;                       // the block solved by the launch before
  const bool chain = blockIdx.x == 0;
  // rows this CTA updates: its block (CTA 0) or 64 rows after it
  const int w0 = u0 + (int)blockIdx.x * kTsNB;
  const int wi = tid >> 2, wq = tid & 3;           // row, part: columns 4 pp + wq
  double cu[16];
  if (b > 0) {
#pragma unroll
    for (int pp = 0; pp < 16; ++pp)
      cu[pp] = (w0 + wi < n) ? T.op(w0 + wi, p0 + 4 * pp + wq) : 0.0;
  }
  // CTA 0: the diagonal block.  Warp 0 holds its first 32 unknowns' matrix,
  // warp 1 the second 32's; every thread 4 entries of the block below the
  // first (row tid >> 3, columns 8 pp + (tid & 7)).
  double d[32], dd = 1.0, rinv = 1.0, cs[4];
  TsForm form = kTsScaled;
  if (chain) {
    if (warp < 2) {
      const int ul = u0 + 32 * warp + lane;
      bool ok = true;
#pragma unroll
      for (int k = 0; k < 32; ++k) {
        const int uk = u0 + 32 * warp + k;
        d[k] = (ul < n && k < lane) ? T.op(ul, uk) : 0.0;
        ok = ok && ts_moderate(d[k], true);
      }
      if (!unit) {
        if (ul < n) dd = T.op(ul, ul);
        ok = ok && ts_moderate(dd, false);
        form = ts_form(n, __all_sync(0xffffffffu, ok));
        if (form != kTsDivide) rinv = 1.0 / dd;
        if (form == kTsScaled) {
#pragma unroll
          for (int k = 0; k < 32; ++k) d[k] *= __shfl_sync(0xffffffffu, rinv, k);
        }
      }
    }
#pragma unroll
    for (int pp = 0; pp < 4; ++pp) {
      const int ur = u0 + 32 + (tid >> 3);
      cs[pp] = (ur < n) ? T.op(ur, u0 + 8 * pp + (tid & 7)) : 0.0;
    }
  }
  pdl_wait();
  pdl_trigger();
  double* mine = (b > 0 && tid < kTsNB) ? &xp[tid] : nullptr;
  if (mine) *mine = xv[T.row(p0 + tid)];
  if (tid >= kTsNB && tid < 2 * kTsNB) {
    const int u = w0 + tid - kTsNB;
    xc[tid - kTsNB] = (u < n) ? xv[T.row(u)] : 0.0;
  }
  __syncthreads();
  if (b > 0) {
    double acc[2] = {0.0, 0.0};
#pragma unroll
    for (int pp = 0; pp < 16; ++pp) acc[pp & 1] = fma(cu[pp], xp[4 * pp + wq], acc[pp & 1]);
    double s = acc[0] + acc[1];
    s += __shfl_xor_sync(0xffffffffu, s, 1);
    s += __shfl_xor_sync(0xffffffffu, s, 2);
    if (wq == 0) {
      const double v = xc[wi] - s;
      if (chain) xc[wi] = v;
      else if (w0 + wi < n) xv[T.row(w0 + wi)] = v;
    }
  }
  if (!chain) return;
  __syncthreads();
  if (warp == 0) {
    const double v = ts_solve32(xc[lane], d, min(32, n - u0), dd, rinv, unit, form);
    xc[lane] = v;
    if (u0 + lane < n) xv[T.row(u0 + lane)] = v;
  }
  if (u0 + 32 >= n) return;                        // uniform
  __syncthreads();
  {
    double s = 0.0;
#pragma unroll
    for (int pp = 0; pp < 4; ++pp) s = fma(cs[pp], xc[8 * pp + (tid & 7)], s);
    s += __shfl_xor_sync(0xffffffffu, s, 1);
    s += __shfl_xor_sync(0xffffffffu, s, 2);
    s += __shfl_xor_sync(0xffffffffu, s, 4);
    if ((tid & 7) == 0) xc[32 + (tid >> 3)] -= s;
  }
  __syncthreads();
  if (warp == 1) {
    const double v = ts_solve32(xc[32 + lane], d, min(32, n - u0 - 32), dd, rinv, unit, form);
    if (u0 + 32 + lane < n) xv[T.row(u0 + 32 + lane)] = v;
  }
}

// Many vectors: a CTA solves V of them from the first block to the last, in shared
// memory.  The four CTAs of an SM are at different places of their chains, so the
// substitutions of one hide behind the updates of others, and there is no launch
// between blocks.  Bound by the FP64 pipe, or by the matrices where each vector has its
// own.  The rows of an update:
//  * kTmRows, no transpose: four lanes to a row, two shuffles;
//  * kTmColumns, a transpose (the rows lie along the lanes) and a matrix that many
//    vectors share, and so find in L2: a thread per row, without shuffles;
//  * kTmSpread, a transpose and few vectors per matrix, which comes from memory: lanes
//    along 32 rows, a part of the columns per warp and all its loads in flight, the parts
//    summed through shared memory; and the next diagonal block's entries on their way
//    during the updates.
// The operations on every element, and their order, are trisolve_step_kernel's.
// Measured, n = 1000 with a transpose, us here (V = 1) and with a launch per block: 300
// vectors 524 and 766, 500 766 and 1155, 1000 1312 and 2102; without one 589 and 765,
// 872 and 1155, 1475 and 2104.  2000 vectors with V = 2: 2446 (V = 1: 2527).  LU solves of
// 1300 systems of n = 300 with a transpose: one right-hand side 578 (four lanes to a row
// 862, a launch per block 733), nine 3477 (a thread per row 4252, a launch per block 5224);
// of one system of n = 2000 with 2000: 17314 with a thread per row, 18365 spread.
constexpr int kTmCtas = 4;
constexpr int kTmShared = 64;       // vectors of one matrix from which it is read from L2
enum TmForm { kTmRows, kTmColumns, kTmSpread };

template <int V, TmForm FORM>
__global__ void __launch_bounds__(kTsThreads, kTmCtas)
trisolve_many_kernel(int n, int nrhs, const double* __restrict__ t, int64_t ldt, int64_t stride_t,
                     int fwd, int unit, double* __restrict__ x, int64_t stride_x) {
  extern __shared__ double ts_x[];                 // V vectors in solve order, zeros past n
  __shared__ double D[2][32][33];                  // the diagonal block's halves, by column
  __shared__ double P[2][FORM == kTmSpread ? V : 1][4][kTsNB];  // partial sums of two tiles
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int nblk = (n + kTsNB - 1) / kTsNB, np = nblk * kTsNB;
  const TsView T{t + (int64_t)blockIdx.y * stride_t, ldt, n, fwd != 0, FORM != kTmRows};
  double* xv = x + (int64_t)blockIdx.y * stride_x + (int64_t)blockIdx.x * V * n;
  const int nv = min(V, nrhs - (int)blockIdx.x * V);
  const int wi = tid >> 2, wq = tid & 3;           // row, part: columns 4 pp + wq
#pragma unroll
  for (int q = 0; q < V; ++q)
    for (int u = tid; u < np; u += kTsThreads)
      ts_x[q * np + u] = (q < nv && u < n) ? xv[(int64_t)q * n + T.row(u)] : 0.0;
  // the halves of block b (warps 0 and 1) on their way to D, a lane's own entries
  auto fetch = [&](int b) {
    const int u1 = b * kTsNB + 32 * warp, m = min(32, n - u1);
#pragma unroll 4
    for (int k = 0; k < m; ++k) {
      const bool in = k < lane && lane < m;
      const unsigned dst = (unsigned)__cvta_generic_to_shared(&D[warp][k][lane]);
      asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(dst),
                   "l"(in ? T.at(u1 + lane, u1 + k) : T.t), "r"(in ? 8 : 0)
                   : "memory");
    }
  };
  if (FORM == kTmSpread && warp < 2) fetch(0);
  for (int b = 0; b < nblk; ++b) {
    const int u0 = b * kTsNB;
    double dd = 1.0, rinv = 1.0, cs[4];
    TsForm form = kTsScaled;
    if (warp < 2) {
      const int ul = u0 + 32 * warp + lane, m = min(32, n - u0 - 32 * warp);
      bool ok = true;
      if (FORM == kTmSpread) asm volatile("cp.async.wait_all;" ::: "memory");
#pragma unroll 8
      for (int k = 0; k < m; ++k) {
        double v;
        if (FORM == kTmSpread) {
          v = D[warp][k][lane];
        } else {
          v = (ul < n && k < lane) ? T.op(ul, u0 + 32 * warp + k) : 0.0;
          D[warp][k][lane] = v;
        }
        ok = ok && ts_moderate(v, true);
      }
      if (!unit) {
        if (ul < n) dd = T.op(ul, ul);
        form = ts_form(n, __all_sync(0xffffffffu, ok && ts_moderate(dd, false)));
        if (form != kTsDivide) rinv = 1.0 / dd;
        if (form == kTsScaled) {
#pragma unroll 8
          for (int k = 0; k < m; ++k) D[warp][k][lane] *= __shfl_sync(0xffffffffu, rinv, k);
        }
      }
    }
#pragma unroll
    for (int pp = 0; pp < 4; ++pp) {
      const int ur = u0 + 32 + (tid >> 3);
      cs[pp] = (ur < n) ? T.op(ur, u0 + 8 * pp + (tid & 7)) : 0.0;
    }
    double* xc = ts_x + u0;
    auto solve = [&](int half) {
      double v[V];
#pragma unroll
      for (int q = 0; q < V; ++q) v[q] = xc[q * np + 32 * half + lane];
      ts_solve32(v, D[half], min(32, n - u0 - 32 * half), dd, rinv, unit, form);
#pragma unroll
      for (int q = 0; q < V; ++q) xc[q * np + 32 * half + lane] = v[q];
    };
    __syncthreads();
    if (warp == 0) solve(0);
    __syncthreads();
    if (u0 + 32 < n) {                             // uniform
#pragma unroll
      for (int q = 0; q < V; ++q) {
        double s = 0.0;
#pragma unroll
        for (int pp = 0; pp < 4; ++pp) s = fma(cs[pp], xc[q * np + 8 * pp + (tid & 7)], s);
        s += __shfl_xor_sync(0xffffffffu, s, 1);
        s += __shfl_xor_sync(0xffffffffu, s, 2);
        s += __shfl_xor_sync(0xffffffffu, s, 4);
        if ((tid & 7) == 0) xc[q * np + 32 + (tid >> 3)] -= s;
      }
      __syncthreads();
      if (warp == 1) solve(1);
      __syncthreads();
    }
    if constexpr (FORM == kTmColumns) {
      for (int u = u0 + kTsNB + tid; u < n; u += kTsThreads) {
        double acc[V][4][2];
#pragma unroll
        for (int q = 0; q < V; ++q)
#pragma unroll
          for (int r = 0; r < 4; ++r) acc[q][r][0] = acc[q][r][1] = 0.0;
#pragma unroll 1
        for (int c = 0; c < kTsNB; c += 16) {
          double cu[16];
#pragma unroll
          for (int e = 0; e < 16; ++e) cu[e] = T.op(u, u0 + c + e);
#pragma unroll
          for (int e = 0; e < 16; ++e)
#pragma unroll
            for (int q = 0; q < V; ++q) {
              double& a = acc[q][e & 3][(e >> 2) & 1];
              a = fma(cu[e], xc[q * np + c + e], a);
            }
        }
#pragma unroll
        for (int q = 0; q < V; ++q)
          ts_x[q * np + u] -= ((acc[q][0][0] + acc[q][0][1]) + (acc[q][1][0] + acc[q][1][1])) +
                              ((acc[q][2][0] + acc[q][2][1]) + (acc[q][3][0] + acc[q][3][1]));
      }
    } else if constexpr (FORM == kTmSpread) {
      if (warp < 2 && b + 1 < nblk) fetch(b + 1);
      const int part = warp & 3, r = 32 * (warp >> 2) + lane;
      for (int w = b + 1; w < nblk; ++w) {
        const int u = w * kTsNB + r;
        double cu[16];
#pragma unroll
        for (int pp = 0; pp < 16; ++pp) cu[pp] = u < n ? T.op(u, u0 + 4 * pp + part) : 0.0;
#pragma unroll
        for (int q = 0; q < V; ++q) {
          double acc[2] = {0.0, 0.0};
#pragma unroll
          for (int pp = 0; pp < 16; ++pp)
            acc[pp & 1] = fma(cu[pp], xc[q * np + 4 * pp + part], acc[pp & 1]);
          P[w & 1][q][part][r] = acc[0] + acc[1];
        }
        __syncthreads();
        if (tid < V * kTsNB) {
          const int q = tid / kTsNB, e = tid % kTsNB;
          const double (&p)[4][kTsNB] = P[w & 1][q];
          ts_x[q * np + w * kTsNB + e] -= (p[0][e] + p[1][e]) + (p[2][e] + p[3][e]);
        }
      }
    } else {
      for (int w = b + 1; w < nblk; ++w) {
        double cu[16];
#pragma unroll
        for (int pp = 0; pp < 16; ++pp)
          cu[pp] = (w * kTsNB + wi < n) ? T.op(w * kTsNB + wi, u0 + 4 * pp + wq) : 0.0;
#pragma unroll
        for (int q = 0; q < V; ++q) {
          double acc[2] = {0.0, 0.0};
#pragma unroll
          for (int pp = 0; pp < 16; ++pp)
            acc[pp & 1] = fma(cu[pp], xc[q * np + 4 * pp + wq], acc[pp & 1]);
          double s = acc[0] + acc[1];
          s += __shfl_xor_sync(0xffffffffu, s, 1);
          s += __shfl_xor_sync(0xffffffffu, s, 2);
          if (wq == 0) ts_x[q * np + w * kTsNB + wi] -= s;
        }
      }
    }
  }
  __syncthreads();
#pragma unroll
  for (int q = 0; q < V; ++q)
    for (int u = tid; u < n; u += kTsThreads)
      if (q < nv) xv[(int64_t)q * n + T.row(u)] = ts_x[q * np + u];
}

// Vectors per CTA of the many-vector solve, 0 where a launch per block is taken: fewer
// vectors than one and a half per SM (n = 1000, 150 vectors: 399 to 452 us against 480;
// n = 4000 4285 to 4718 against 4390), or a matrix whose triangle the L2 cache may not
// hold, since every CTA reads all of it.
// Two per CTA above eight per SM, and where one each is more than the SMs take at once
// but two each are not, for small n, whose second round is the longer part (us with one
// and two, 1000 vectors: n = 200 177 and 142, 700 774 and 721, 1000 1312 and 1442; 700
// vectors: n = 1000 1280 and 1060, 2000 3360 and 3870).
constexpr int kTmMaxN = 4096;

static int ts_many(int64_t batch, int n, int nrhs) {
  const int64_t vectors = batch * nrhs;
  if (n > kTmMaxN || 2 * vectors < 3 * sm_count()) return 0;
  const int64_t per_sm = (vectors + sm_count() - 1) / sm_count();
  const bool two = per_sm > 8 || (per_sm > kTmCtas && n <= (per_sm <= 6 ? 1024 : 768));
  // (a system's odd vector has a CTA of its own: no loss among eight or more)
  return two && (nrhs % 2 == 0 || nrhs >= 8) ? 2 : 1;
}

// The whole solve in one launch for n up to 64 kTcMaxBlocks: a cluster of C CTAs
// per vector, CTA r holding the blocks r, r + C, ... of x in shared memory.  Step
// b + 1: its owner subtracts x_b from its block, solves it and writes x_{b+1} into
// every CTA's shared memory; then, and in the other CTAs meanwhile, x_b is
// subtracted from the later blocks.  Matrix entries of the chain are loaded before
// the wait for x_b.  A CTA arrives at the cluster barrier of step b + 1 before its
// own later blocks' updates, so it may lag behind the chain by a step or two (four
// buffers of x; program order keeps a buffer's last read before the arrival that
// lets it be overwritten).  The operations on every element, and their order, are
// trisolve_step_kernel's.
// Measured (one vector, us): n = 401 60, 1000 126, 1531 185, 2003 246, against 69, 135,
// 217 and 282 with a launch per block (five or more vectors), whose hand-over it saves;
// the chain of a block (two substitutions, the update, the push and the barrier)
// remains.
constexpr int kTcMaxBlocks = 32;
constexpr int kTcMax = 16;

__global__ void __launch_bounds__(kTsThreads, 1)
trisolve_cluster_kernel(int n, const double* __restrict__ t, int64_t ldt, int64_t stride_t,
                        int fwd, int trans, int unit, double* __restrict__ x, int64_t stride_x) {
  __shared__ double xs[kTcMaxBlocks / kTcMax][kTsNB];  // this CTA's blocks, in turn
  __shared__ double xb[4][kTsNB];              // solved blocks, written by their owners
  cg::cluster_group cluster = cg::this_cluster();
  const int C = (int)cluster.num_blocks(), rank = (int)cluster.block_rank();
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int nblk = (n + kTsNB - 1) / kTsNB;
  const TsView T{t + (int64_t)blockIdx.z * stride_t, ldt, n, fwd != 0, trans != 0};
  double* xv = x + (int64_t)blockIdx.z * stride_x + (int64_t)blockIdx.y * n;
  const int wi = tid >> 2, wq = tid & 3;           // row, part: columns 4 pp + wq
  double cu[16], d[32], dd = 1.0, rinv = 1.0, cs[4];
  TsForm form = kTsScaled;                         // (two blocks and more)
  auto load_update = [&](int w, int b) {
#pragma unroll
    for (int pp = 0; pp < 16; ++pp)
      cu[pp] = (w * kTsNB + wi < n) ? T.op(w * kTsNB + wi, b * kTsNB + 4 * pp + wq) : 0.0;
  };
  auto update = [&](double* xw, const double* xp) {
    double acc[2] = {0.0, 0.0};
#pragma unroll
    for (int pp = 0; pp < 16; ++pp) acc[pp & 1] = fma(cu[pp], xp[4 * pp + wq], acc[pp & 1]);
    double s = acc[0] + acc[1];
    s += __shfl_xor_sync(0xffffffffu, s, 1);
    s += __shfl_xor_sync(0xffffffffu, s, 2);
    if (wq == 0) xw[wi] -= s;
  };
  auto load_diag = [&](int b) {
    const int u0 = b * kTsNB;
    form = kTsScaled;
    dd = rinv = 1.0;
    if (warp < 2) {
      const int ul = u0 + 32 * warp + lane;
      bool ok = true;
#pragma unroll
      for (int k = 0; k < 32; ++k) {
        const int uk = u0 + 32 * warp + k;
        d[k] = (ul < n && k < lane) ? T.op(ul, uk) : 0.0;
      }
      if (!unit && ul < n) dd = T.op(ul, ul);
      if (!unit) {
#pragma unroll
        for (int k = 0; k < 32; ++k) ok = ok && ts_moderate(d[k], true);
        ok = ok && ts_moderate(dd, false);
        form = ts_form(n, __all_sync(0xffffffffu, ok));
        if (form != kTsDivide) rinv = 1.0 / dd;
        if (form == kTsScaled) {
#pragma unroll
          for (int k = 0; k < 32; ++k) d[k] *= __shfl_sync(0xffffffffu, rinv, k);
        }
      }
    }
#pragma unroll
    for (int pp = 0; pp < 4; ++pp) {
      const int ur = u0 + 32 + (tid >> 3);
      cs[pp] = (ur < n) ? T.op(ur, u0 + 8 * pp + (tid & 7)) : 0.0;
    }
  };
  // block b solved in place in xc, out to memory and to every CTA's buffer
  auto solve = [&](double* xc, int b) {
    const int u0 = b * kTsNB;
    if (warp == 0) xc[lane] = ts_solve32(xc[lane], d, 32, dd, rinv, unit, form);
    __syncthreads();
    double s = 0.0;
#pragma unroll
    for (int pp = 0; pp < 4; ++pp) s = fma(cs[pp], xc[8 * pp + (tid & 7)], s);
    s += __shfl_xor_sync(0xffffffffu, s, 1);
    s += __shfl_xor_sync(0xffffffffu, s, 2);
    s += __shfl_xor_sync(0xffffffffu, s, 4);
    if ((tid & 7) == 0) xc[32 + (tid >> 3)] -= s;
    __syncthreads();
    if (warp == 1) xc[32 + lane] = ts_solve32(xc[32 + lane], d, 32, dd, rinv, unit, form);
    __syncthreads();
    const double v = xc[tid & (kTsNB - 1)];
#pragma unroll
    for (int q = 0; q < kTcMax / 4; ++q) {
      const int dst = 4 * q + (tid >> 6);
      if (dst < C) *cluster.map_shared_rank(&xb[b & 3][tid & (kTsNB - 1)], dst) = v;
    }
    if (tid < kTsNB && u0 + tid < n) xv[T.row(u0 + tid)] = v;
  };
  for (int e = tid; rank + (e / kTsNB) * C < nblk; e += kTsThreads) {
    const int u = (rank + (e / kTsNB) * C) * kTsNB + e % kTsNB;
    xs[e / kTsNB][e % kTsNB] = (u < n) ? xv[T.row(u)] : 0.0;
  }
  cluster.sync();                                  // all run before any remote store
  if (rank == 0) {
    load_diag(0);
    solve(xs[0], 0);
  }
  cluster.barrier_arrive();
  for (int b = 0; b + 1 < nblk; ++b) {
    const bool next = rank == (b + 1) % C;
    if (next) {
      load_diag(b + 1);
      load_update(b + 1, b);
    }
    cluster.barrier_wait();                        // x_b is here
    const double* xp = xb[b & 3];
    if (next) {
      double* xc = xs[(b + 1) / C];
      update(xc, xp);
      __syncthreads();
      solve(xc, b + 1);
    }
    cluster.barrier_arrive();
    // this CTA's blocks after b + 1
    for (int w = rank + ((b + 2 - rank + C - 1) / C) * C; w < nblk; w += C) {
      load_update(w, b);
      update(xs[w / C], xp);
    }
  }
  cluster.barrier_wait();  // no CTA leaves while another may still write its shared memory
}

// CTAs per vector of the one-launch solve, 0 where a launch per block is taken:
// n above its blocks (two per CTA: more of them would hold up the chain) or one
// block, more vectors than clusters fit on the SMs at once, or no cluster to be
// had.  us at n = 1000 here and with a launch per block: 4 vectors 120 and 132, 8
// vectors 231 and 138 (the clusters run one after the other).
static int ts_cluster_size(int64_t vectors, int n) {
  const int nblk = (n + kTsNB - 1) / kTsNB;
  if (nblk < 2 || nblk > kTcMaxBlocks) return 0;
  const int c = nblk < kTcMax ? nblk : kTcMax;
  int room = kTcMax;                 // SMs of one processing cluster that it takes
  while (room / 2 >= c) room /= 2;
  if (vectors * room > 4 * kTcMax) return 0;
  return cluster_fits(reinterpret_cast<const void*>(trisolve_cluster_kernel), c, kTsThreads, 0) ? c : 0;
}

int trisolve_blocked(int64_t batch, int n, int nrhs, const double* t, int64_t ldt,
                     int64_t stride_t, int lower, int trans, int unit, double* x,
                     int64_t stride_x, cudaStream_t st) {
  const int fwd = (lower != 0) != (trans != 0);
  const int nblk = (n + kTsNB - 1) / kTsNB;
  const int c = ts_cluster_size(batch * nrhs, n);
  if (c > 0) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)c, (unsigned)nrhs, (unsigned)batch);
    cfg.blockDim = dim3(kTsThreads);
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = (unsigned)c;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    LXGB_CUDA_TRY(cudaLaunchKernelEx(&cfg, trisolve_cluster_kernel, n, t, ldt, stride_t, fwd, trans,
                                     unit, x, stride_x),
                  "trisolve: launch");
    return check_launch("trisolve");
  }
  if (const int v = ts_many(batch, n, nrhs)) {
    auto fn = v == 2 ? trisolve_many_kernel<2, kTmRows> : trisolve_many_kernel<1, kTmRows>;
    if (trans && nrhs >= kTmShared)
      fn = v == 2 ? trisolve_many_kernel<2, kTmColumns> : trisolve_many_kernel<1, kTmColumns>;
    else if (trans)
      fn = v == 2 ? trisolve_many_kernel<2, kTmSpread> : trisolve_many_kernel<1, kTmSpread>;
    const size_t smem = (size_t)v * nblk * kTsNB * sizeof(double);
    LXGB_CUDA_TRY(ensure_dynamic_smem(reinterpret_cast<const void*>(fn), (int)smem),
                  "trisolve: set smem");
    fn<<<dim3((unsigned)((nrhs + v - 1) / v), (unsigned)batch), kTsThreads, smem, st>>>(
        n, nrhs, t, ldt, stride_t, fwd, unit, x, stride_x);
    return check_launch("trisolve");
  }
  for (int b = 0; b < nblk; ++b) {
    const int after = n - (b + 1) * kTsNB;         // rows after this block
    const unsigned gx = 1u + (unsigned)((b > 0 && after > 0) ? (after + kTsNB - 1) / kTsNB : 0);
    const dim3 grid(gx, (unsigned)nrhs, (unsigned)batch);
    if (b == 0) {
      // not a dependent launch: the kernel before it may still write the matrix
      trisolve_step_kernel<<<grid, kTsThreads, 0, st>>>(n, t, ldt, stride_t, fwd, trans, unit, b,
                                                        x, stride_x);
    } else {
      LXGB_CUDA_TRY(launch_pdl(trisolve_step_kernel, grid, dim3(kTsThreads), 0, st, 1, n, t, ldt,
                               stride_t, fwd, trans, unit, b, x, stride_x),
                    "trisolve: launch");
    }
  }
  return check_launch("trisolve");
}

}  // namespace lxgb
