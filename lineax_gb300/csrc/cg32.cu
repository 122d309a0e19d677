// Mixed-precision CG for the 5-point Poisson operator, k right-hand sides:
// the iteration vectors p, r, Ap and the running correction x_lo are FP32
// (the HBM stream of the hot loop), the solution x and the right-hand side b
// FP64.  Every `check` iterations (16 by default) the host calls lxgb_cg32_refresh, which
// folds x_lo into x in FP64, recomputes the true residual r = b - A x in FP64
// (residual replacement: the recurrence residual restarts from it, the search
// direction is kept), evaluates lineax's stopping test on that true residual
// (max_i |r_i| / (atol + rtol |b_i|) <= 1, lineax/_solver/cg.py:149-160) and
// resets gamma = rᵀr.  Between refreshes an iteration is
//   alpha = gamma / <p, Ap>    (lineax's breakdown guard)
//   x_lo += alpha p, r -= alpha Ap, <r, r>
//   beta = <r, r> / gamma, p = r + beta p
// in two passes over memory, both bound by HBM:
//   c32_residual_kernel: A p again from p (a stencil, five operations), r and
//     <r, r>: 12 bytes per point;
//   c32_step_kernel: x_lo with the old p, the new p, and <p, Ap> of the new p
//     from a tile in shared memory: 20 bytes per point.  It writes the new p to
//     the other of two buffers, since neighbouring CTAs read the old one.
// A p itself is never stored.  (Ap stored and every update a pass of its own:
// 44 bytes per point.)
// Dot products accumulate FP32 products in FP32 over a thread's few elements
// and combine the per-thread sums in FP64, in a fixed order.  Each right-hand
// side carries its own flags; an inactive one is left untouched, so results do
// not depend on the other right-hand sides in the block.
#include <math.h>

#include "common.cuh"

namespace lxgb {

constexpr int kC32Threads = 256;
constexpr int kC32RowsPerCta = 16;  // grid rows per CTA of the stencil pass
constexpr int kC32MaxParts = 1024;  // partial sums per right-hand side

struct C32State {
  double* gamma;   // k: <r, r> of the current recurrence
  double* alpha;   // k
  double* beta;    // k
  int* act;        // k: not finished (the next refresh still folds x_lo)
  int* run;        // k: iterating
  int* steps;      // k
  int* conv;       // k: 1 converged, 2 breakdown or NaN test
  double* part;    // k * kC32MaxParts partial sums
};

static int64_t c32_state_bytes(int k) {
  return 256 + (int64_t)k * (3 * 8 + 4 * 4) + 256 + (int64_t)k * kC32MaxParts * 8;
}

static C32State c32_carve(void* work, int k) {
  C32State s;
  char* p = reinterpret_cast<char*>(work) + 256;
  s.gamma = reinterpret_cast<double*>(p); p += (int64_t)k * 8;
  s.alpha = reinterpret_cast<double*>(p); p += (int64_t)k * 8;
  s.beta = reinterpret_cast<double*>(p); p += (int64_t)k * 8;
  s.act = reinterpret_cast<int*>(p); p += (int64_t)k * 4;
  s.run = reinterpret_cast<int*>(p); p += (int64_t)k * 4;
  s.steps = reinterpret_cast<int*>(p); p += (int64_t)k * 4;
  s.conv = reinterpret_cast<int*>(p); p += (int64_t)k * 4;
  p = reinterpret_cast<char*>(((uintptr_t)p + 255) & ~(uintptr_t)255);
  s.part = reinterpret_cast<double*>(p);
  return s;
}

__device__ __forceinline__ double c32_block_sum(double v, double* sm) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  v = warp_sum(v);
  if (lane == 0) sm[warp] = v;
  __syncthreads();
  double t = 0.0;
  if (threadIdx.x == 0)
    for (int w = 0; w < (int)(blockDim.x >> 5); ++w) t += sm[w];
  return t;
}

// Partial count for the stencil pass over an nx×ny grid.
static int c32_parts(int64_t nx, int64_t ny) {
  return (int)(((ny + kC32Threads - 1) / kC32Threads) *
               ((nx + kC32RowsPerCta - 1) / kC32RowsPerCta));
}

// p' = r + beta p written to pnew, x_lo += alpha p (STEP), and the partials of
// <p', A p'>; without STEP only the partials of <p, A p> (the first iteration
// after a refresh).  One CTA takes 256 columns and 16 rows: its 18 x 258 points
// of p' go to shared memory with 16-byte loads (VEC = 4: ny a multiple of four
// and all pointers on 16 bytes; one float at a time otherwise), then one thread
// per column walks the rows, so a thread's sum has the same terms in the same
// order whatever VEC is.
// Bound by HBM.  Measured at 2048 x 2048, 64 right-hand sides: 761 us, 7.0 TB/s of these
// 20 bytes.  That is 3 % above a plain copy's rate (6.79): three bytes are read for two
// written, and L2 may still hold a part of p and r.  (The passes it replaces, a stencil
// with A p stored, p and half of the update: 847, 584 and about 620 us.)
template <bool STEP, int VEC>
__global__ void __launch_bounds__(kC32Threads)
c32_step_kernel(int64_t nx, int64_t ny, C32State s, const float* __restrict__ r,
                const float* __restrict__ p, float* __restrict__ pnew, float* __restrict__ xlo) {
  constexpr int kRows = kC32RowsPerCta + 2;
  constexpr int kPerRow = kC32Threads / VEC;            // threads on one row
  constexpr int kStep = kC32Threads / kPerRow;          // rows at a time
  constexpr int kIts = (kRows + kStep - 1) / kStep;
  constexpr int kBatch = VEC == 4 ? 3 : 6;           // loads in flight per thread and array
  __shared__ __align__(16) float T[kRows][kC32Threads + 8];
  __shared__ double sm[kC32Threads / 32];
  pdl_wait();
  const int c = blockIdx.z;
  const int part = blockIdx.y * gridDim.x + blockIdx.x;
  if (!s.run[c]) return;  // uniform per CTA
  const int64_t n = nx * ny;
  const float* pc = p + (int64_t)c * n;
  const float* rc = r + (int64_t)c * n;
  const float al = STEP ? (float)s.alpha[c] : 0.0f, be = STEP ? (float)s.beta[c] : 0.0f;
  const int tid = threadIdx.x;
  const int64_t j0 = (int64_t)blockIdx.x * kC32Threads, i0 = (int64_t)blockIdx.y * kC32RowsPerCta;
  const int rr = tid / kPerRow, cc = (tid % kPerRow) * VEC;
  struct alignas(4 * VEC) Pack { float v[VEC]; };
#pragma unroll
  for (int h = 0; h < kIts; h += kBatch) {  // (rows past the tile are masked)
    Pack vp[kBatch], vr[kBatch], vx[kBatch];
#pragma unroll
    for (int u = 0; u < kBatch; ++u) {
      const int row = (h + u) * kStep + rr;
      const int64_t i = i0 - 1 + row, o = i * ny + j0 + cc;
      const bool in = row < kRows && i >= 0 && i < nx && j0 + cc < ny;
      const bool own = in && row >= 1 && row <= kC32RowsPerCta;
#pragma unroll
      for (int q = 0; q < VEC; ++q) vp[u].v[q] = vr[u].v[q] = vx[u].v[q] = 0.0f;
      if (in) vp[u] = *reinterpret_cast<const Pack*>(pc + o);
      if (STEP && in) vr[u] = *reinterpret_cast<const Pack*>(rc + o);
      if (STEP && own) vx[u] = *reinterpret_cast<const Pack*>(xlo + (int64_t)c * n + o);
    }
#pragma unroll
    for (int u = 0; u < kBatch; ++u) {
      const int row = (h + u) * kStep + rr;
      const int64_t i = i0 - 1 + row, o = i * ny + j0 + cc;
      const bool in = row < kRows && i >= 0 && i < nx && j0 + cc < ny;
      const bool own = in && row >= 1 && row <= kC32RowsPerCta;
      Pack w = vp[u];
      if (STEP && in) {
#pragma unroll
        for (int q = 0; q < VEC; ++q) {
          w.v[q] = fmaf(be, vp[u].v[q], vr[u].v[q]);
          vx[u].v[q] = fmaf(al, vp[u].v[q], vx[u].v[q]);
        }
        if (own) {
          *reinterpret_cast<Pack*>(pnew + (int64_t)c * n + o) = w;
          *reinterpret_cast<Pack*>(xlo + (int64_t)c * n + o) = vx[u];
        }
      }
      if (row < kRows) *reinterpret_cast<Pack*>(&T[row][4 + cc]) = w;
    }
  }
  // the columns left and right of the tile
  if (tid < 2 * kRows) {
    const int row = tid >> 1, right = tid & 1;
    const int64_t i = i0 - 1 + row, j = right ? j0 + kC32Threads : j0 - 1;
    float w = 0.0f;
    if (i >= 0 && i < nx && j >= 0 && j < ny) {
      w = pc[i * ny + j];
      if (STEP) w = fmaf(be, w, rc[i * ny + j]);
    }
    T[row][right ? 4 + kC32Threads : 3] = w;
  }
  __syncthreads();
  float acc = 0.0f;
  if (j0 + tid < ny) {
    const int rows = (int)min((int64_t)kC32RowsPerCta, nx - i0);
    float up = T[0][4 + tid], cen = T[1][4 + tid];
#pragma unroll 8
    for (int i = 1; i <= rows; ++i) {
      const float dn = T[i + 1][4 + tid], lf = T[i][3 + tid], rt = T[i][5 + tid];
      const float v = fmaf(4.0f, cen, -((up + dn) + (lf + rt)));
      acc = fmaf(cen, v, acc);
      up = cen;
      cen = dn;
    }
  }
  const double t = c32_block_sum((double)acc, sm);
  if (tid == 0) s.part[(int64_t)c * kC32MaxParts + part] = t;
}

// Sum of vector c's partials in index order (one warp per right-hand side).
__device__ double c32_combine(const double* part, int P) {
  const int lane = threadIdx.x & 31;
  double v = 0.0;
#pragma unroll 16
  for (int i = lane; i < P; i += 32) v += part[i];
  return warp_sum(v);
}

// alpha = gamma / <p, Ap>; a non-positive or non-finite curvature stops the
// right-hand side (breakdown, as lineax's NaN alpha at cg.py:172-178).
__global__ void c32_alpha_kernel(int k, C32State s, int P) {
  pdl_wait();
  const int c = blockIdx.x;
  if (!s.run[c]) return;
  const double pap = c32_combine(s.part + (int64_t)c * kC32MaxParts, P);
  if (threadIdx.x == 0) {
    const double a = s.gamma[c] / pap;
    if (!(pap > 0.0) || !isfinite(a)) {
      s.run[c] = 0;  // the next refresh folds x_lo and ends this right-hand side
      s.conv[c] = 2;
    }
    s.alpha[c] = a;
  }
}

// r -= alpha A p and the partials of <r, r>.  Partial b (of P) sums the points
// b * 256 + t + m * 256 P, t < 256, each t's over m first.  A CTA forms G
// neighbouring partials, so for one m it reads 256 G consecutive points and the
// rows around them: the values above, below, left and right are found in L1,
// except one row at each end.  Measured at 2048 x 2048, 64 right-hand sides (12
// bytes per point, 450 us at HBM's rate): one partial per CTA, three rows read
// from L2 for one updated, 759 us; G = 32 643; with the next points prefetched
// into L2 540; G = 16 523.
constexpr int kC32ResThreads = 512;

template <int G>
__global__ void __launch_bounds__(kC32ResThreads, 2)
c32_residual_kernel(int n, int ny, int P, C32State s, const float* __restrict__ p,
                    float* __restrict__ r) {
  constexpr int kS = G / 2, kU = kS < 4 ? kS : 4;
  __shared__ double sm[G][kC32Threads / 32];
  pdl_wait();
  const int c = blockIdx.y;
  if (!s.run[c]) return;
  const float a = (float)s.alpha[c];
  const float* pc = p + (int64_t)c * n;
  float* rc = r + (int64_t)c * n;
  const int tid = threadIdx.x, b0 = blockIdx.x * G;
  const int stride = P * kC32Threads;
  const int ends = min(stride, (b0 + G) * kC32Threads);  // of this CTA's points at m = 0
  const int dcol = kC32ResThreads % ny;
  float acc[kS];
#pragma unroll
  for (int q = 0; q < kS; ++q) acc[q] = 0.0f;
  for (int m = 0; m < n; m += stride) {
    const int o0 = b0 * kC32Threads + tid + m, last = min(n, m + ends);
    if (o0 - tid >= n) break;
    // the next m's lines into L2: the loads below keep too few bytes in flight
    // to cover the latency of HBM
    for (int w = tid; w < 2 * G * kC32Threads / 32; w += kC32ResThreads) {
      const bool pr = w >= G * kC32Threads / 32;
      const int o = o0 - tid + stride + 32 * (pr ? w - G * kC32Threads / 32 : w);
      if (o < n) asm volatile("prefetch.global.L2 [%0];" ::"l"((pr ? rc : pc) + o));
    }
    int col = o0 % ny;
#pragma unroll
    for (int h = 0; h < kS; h += kU) {
      float cen[kU], up[kU], dn[kU], lf[kU], rt[kU], rv[kU];
#pragma unroll
      for (int u = 0; u < kU; ++u) {
        const int o = o0 + (h + u) * kC32ResThreads;
        const bool in = o < last;
        cen[u] = in ? pc[o] : 0.0f;
        up[u] = (in && o >= ny) ? pc[o - ny] : 0.0f;
        dn[u] = (in && o + ny < n) ? pc[o + ny] : 0.0f;
        lf[u] = (in && col > 0) ? pc[o - 1] : 0.0f;
        rt[u] = (in && col + 1 < ny) ? pc[o + 1] : 0.0f;
        rv[u] = in ? rc[o] : 0.0f;
        col += dcol;
        if (col >= ny) col -= ny;
      }
#pragma unroll
      for (int u = 0; u < kU; ++u) {
        const int o = o0 + (h + u) * kC32ResThreads;
        if (o < last) {
          const float v = fmaf(4.0f, cen[u], -((up[u] + dn[u]) + (lf[u] + rt[u])));
          const float rn = fmaf(-a, v, rv[u]);
          rc[o] = rn;
          acc[h + u] = fmaf(rn, rn, acc[h + u]);
        }
      }
    }
  }
#pragma unroll
  for (int q = 0; q < kS; ++q) {
    const double t = warp_sum((double)acc[q]);
    if ((tid & 31) == 0) sm[2 * q + (tid >> 8)][(tid >> 5) & 7] = t;
  }
  __syncthreads();
  if (tid < G && b0 + tid < P) {
    double t = 0.0;
#pragma unroll
    for (int w = 0; w < kC32Threads / 32; ++w) t += sm[tid][w];
    s.part[(int64_t)c * kC32MaxParts + b0 + tid] = t;
  }
}

// beta = <r, r> / gamma, gamma = <r, r>, steps += 1 (one warp per right-hand side).
__global__ void c32_beta_kernel(int k, C32State s, int P) {
  pdl_wait();
  const int c = blockIdx.x;
  if (!s.run[c]) return;
  const double rr = c32_combine(s.part + (int64_t)c * kC32MaxParts, P);
  if (threadIdx.x == 0) {
    s.beta[c] = rr / s.gamma[c];
    s.gamma[c] = rr;
    s.steps[c] += 1;
  }
}

// x_lo += alpha p, p' = r + beta p (the last iteration before a refresh; pnew
// may be p).
template <int VEC>
__global__ void __launch_bounds__(kC32Threads)
c32_direction_kernel(int64_t n, C32State s, const float* __restrict__ r, const float* p,
                     float* pnew, float* __restrict__ xlo) {
  struct alignas(4 * VEC) Pack { float v[VEC]; };
  pdl_wait();
  const int c = blockIdx.y;
  if (!s.run[c]) return;
  const float al = (float)s.alpha[c], be = (float)s.beta[c];
  const Pack* rq = reinterpret_cast<const Pack*>(r + (int64_t)c * n);
  const Pack* pq = reinterpret_cast<const Pack*>(p + (int64_t)c * n);
  Pack* nq = reinterpret_cast<Pack*>(pnew + (int64_t)c * n);
  Pack* xq = reinterpret_cast<Pack*>(xlo + (int64_t)c * n);
  const int64_t nq4 = n / VEC;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < nq4;
       i += (int64_t)gridDim.x * blockDim.x) {
    const Pack pv = pq[i], rv = rq[i];
    Pack xv = xq[i], w;
#pragma unroll
    for (int q = 0; q < VEC; ++q) {
      xv.v[q] = fmaf(al, pv.v[q], xv.v[q]);
      w.v[q] = fmaf(be, pv.v[q], rv.v[q]);
    }
    xq[i] = xv;
    nq[i] = w;
  }
}

// (float)v, rounded to nearest even, on integers where the result is a normal
// number or zero: the FP64 pipe, which also converts, bounds the refresh.
__device__ __forceinline__ float c32_to_float(double v) {
  const uint32_t hi = (uint32_t)__double2hiint(v), lo = (uint32_t)__double2loint(v);
  const uint32_t e = (hi >> 20) & 0x7FFu, sign = hi & 0x80000000u;
  if (e - 897u < 253u) {  // 2^-126 <= |v| < 2^127
    uint32_t f = ((e - 896u) << 23) | ((hi & 0xFFFFFu) << 3) | (lo >> 29);
    const uint32_t rest = lo & 0x1FFFFFFFu;
    f += (rest + (f & 1u) > 0x10000000u) ? 1u : 0u;
    return __uint_as_float(f | sign);
  }
  if ((hi & 0x7FFFFFFFu) == 0 && lo == 0) return __uint_as_float(sign);
  return (float)v;
}

// |v| / s against 1 without a division: 0 (<= 1), 1 (> 1), 2 (NaN).
__device__ __forceinline__ int c32_ratio_code(double v, double sc) {
  const long long kInf = 0x7FF0000000000000LL;
  const long long av = __double_as_longlong(v) & 0x7FFFFFFFFFFFFFFFLL;
  const long long sb = __double_as_longlong(sc);
  const long long as = sb & 0x7FFFFFFFFFFFFFFFLL;
  if (av > kInf || as > kInf) return 2;
  if (as == 0) return av == 0 ? 2 : 1;
  if (as == kInf) return av == kInf ? 2 : 0;
  if (sb < 0) return 0;
  return av > sb ? 1 : 0;
}

// Refresh, first pass (active right-hand sides): x += x_lo, x_lo = 0.  VEC = 4
// where both are on 16 bytes: 0.99 ms against 1.10 one by one at 2048 x 2048, 64
// right-hand sides (24 bytes per point).
template <int VEC>
__global__ void __launch_bounds__(kC32Threads)
c32_fold_kernel(int64_t n, C32State s, double* __restrict__ x, float* __restrict__ xlo) {
  struct alignas(VEC == 4 ? 16 : 8) Two { double v[VEC == 4 ? 2 : 1]; };
  struct alignas(4 * VEC) Pack { float v[VEC]; };
  const int c = blockIdx.y;
  if (!s.act[c]) return;
  Two* xq = reinterpret_cast<Two*>(x + (int64_t)c * n);
  Pack* lq = reinterpret_cast<Pack*>(xlo + (int64_t)c * n);
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n / VEC;
       i += (int64_t)gridDim.x * blockDim.x) {
    const Pack l = lq[i];
    Pack zero;
#pragma unroll
    for (int q = 0; q < VEC; ++q) zero.v[q] = 0.0f;
    if (VEC == 4) {
      Two a = xq[2 * i], b = xq[2 * i + 1];
      a.v[0] += (double)l.v[0];
      a.v[VEC / 4] += (double)l.v[VEC / 4];
      b.v[0] += (double)l.v[VEC / 2];
      b.v[VEC / 4] += (double)l.v[VEC - 1];
      xq[2 * i] = a;
      xq[2 * i + 1] = b;
    } else {
      Two a = xq[i];
      a.v[0] += (double)l.v[0];
      xq[i] = a;
    }
    lq[i] = zero;
  }
}

// Refresh, second pass: r = b - A x in FP64 (stored as FP32), partial <r, r>
// and the stopping-test code per CTA.  Bound by the FP64 pipe (five operations
// per point; six where the stopping test needs its tolerance).  Measured at
// 2048 x 2048, 64 right-hand sides: 3.04 ms (4.72 with the conversion and the
// tolerance of every point on that pipe).
__global__ void __launch_bounds__(kC32Threads)
c32_refresh_kernel(int64_t nx, int64_t ny, C32State s, const double* __restrict__ b,
                   const double* __restrict__ x, float* __restrict__ r,
                   int* __restrict__ codes, double rtol, double atol) {
  __shared__ double sm[kC32Threads / 32];
  __shared__ int s_code;
  const int c = blockIdx.z;
  const int part = blockIdx.y * gridDim.x + blockIdx.x;
  if (!s.act[c]) return;
  const int64_t n = nx * ny;
  const double* xc = x + (int64_t)c * n;
  const int64_t j = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (threadIdx.x == 0) s_code = 0;
  __syncthreads();
  const int64_t i0 = (int64_t)blockIdx.y * kC32RowsPerCta;
  const int64_t i1 = min(nx, i0 + kC32RowsPerCta);
  constexpr int kU = 4;
  const bool plain = atol > 0.0 && atol < 1e100 && rtol >= 0.0 && rtol < 1e100;
  float acc = 0.0f;
  int code = 0;
  if (j < ny) {
    const double* bc = b + (int64_t)c * n;
    float* rc = r + (int64_t)c * n;
    double up = (i0 > 0) ? xc[(i0 - 1) * ny + j] : 0.0;
    double cen = xc[i0 * ny + j];
    for (int64_t ib = i0; ib < i1; ib += kU) {
      double dn[kU], lf[kU], rt[kU], bv[kU];
#pragma unroll
      for (int u = 0; u < kU; ++u) {
        const int64_t i = ib + u, o = i * ny + j;
        const bool in = i < i1;
        dn[u] = (in && i + 1 < nx) ? xc[o + ny] : 0.0;
        lf[u] = (in && j > 0) ? xc[o - 1] : 0.0;
        rt[u] = (in && j + 1 < ny) ? xc[o + 1] : 0.0;
        bv[u] = in ? bc[o] : 0.0;
      }
#pragma unroll
      for (int u = 0; u < kU; ++u) {
        if (ib + u >= i1) break;
        const double ax = fma(4.0, cen, -((up + dn[u]) + (lf[u] + rt[u])));
        const double rv = bv[u] - ax;
        const float rf = c32_to_float(rv);
        rc[(ib + u) * ny + j] = rf;
        acc = fmaf(rf, rf, acc);
        // Once a point is above its tolerance only a NaN quotient can change
        // the thread's code, and with a tolerance in [atol, 2^1000] (`plain`,
        // |b| < 2^512) and a finite residual there is none.
        const uint32_t eb = ((uint32_t)__double2hiint(bv[u]) >> 20) & 0x7FFu;
        const uint32_t er = ((uint32_t)__double2hiint(rv) >> 20) & 0x7FFu;
        if (code == 0 || !plain || eb >= 1023u + 512u || er == 0x7FFu)
          code = max(code, c32_ratio_code(rv, fma(rtol, fabs(bv[u]), atol)));
        up = cen;
        cen = dn[u];
      }
    }
  }
  const double t = c32_block_sum((double)acc, sm);
  if (code) atomicMax(&s_code, code);
  __syncthreads();
  if (threadIdx.x == 0) {
    s.part[(int64_t)c * kC32MaxParts + part] = t;
    codes[(int64_t)c * kC32MaxParts + part] = s_code;
  }
}

// gamma = <r, r> of the replaced residual; the right-hand side ends when the
// test passes (max code 0), when it is NaN (lineax: a NaN norm ends the
// loop), after a breakdown, or at max_steps.
__global__ void c32_refresh_final_kernel(int k, C32State s, const int* __restrict__ codes, int P,
                                         int64_t max_steps) {
  const int c = blockIdx.x;
  if (!s.act[c]) return;
  const double rr = c32_combine(s.part + (int64_t)c * kC32MaxParts, P);
  const int lane = threadIdx.x & 31;
  int m = 0;
  for (int i = lane; i < P; i += 32) m = max(m, codes[(int64_t)c * kC32MaxParts + i]);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) m = max(m, __shfl_xor_sync(0xffffffffu, m, o));
  if (threadIdx.x == 0) {
    s.gamma[c] = rr;
    if (s.conv[c] == 2) {
      s.act[c] = s.run[c] = 0;
    } else if (m != 1) {
      s.act[c] = s.run[c] = 0;
      s.conv[c] = (m == 0) ? 1 : 2;
    } else if (s.steps[c] >= max_steps) {
      s.act[c] = s.run[c] = 0;
    }
  }
}

__global__ void c32_init_kernel(int k, C32State s, int64_t max_steps) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= k) return;
  s.act[c] = 1;
  s.run[c] = max_steps > 0 ? 1 : 0;
  s.steps[c] = 0;
  s.conv[c] = 0;
  s.gamma[c] = 0.0;
}

__global__ void c32_status_kernel(int k, C32State s, int32_t* out) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= k) return;
  out[3 * c] = s.act[c];
  out[3 * c + 1] = s.steps[c];
  out[3 * c + 2] = s.conv[c];  // 0: max steps (or running), 1 converged, 2 breakdown / NaN
}

}  // namespace lxgb

using namespace lxgb;

extern "C" int64_t lxgb_cg32_workspace_size(int32_t nrhs) {
  // state + partial codes
  return c32_state_bytes(nrhs > 0 ? nrhs : 1) + (int64_t)(nrhs > 0 ? nrhs : 1) * kC32MaxParts * 4 +
         256;
}

static int c32_check(int32_t k, int64_t nx, int64_t ny, void* work, int64_t wbytes) {
  LXGB_REQUIRE(k >= 1 && k <= 65535 && nx >= 1 && ny >= 1, "cg32: bad sizes");
  LXGB_REQUIRE(nx <= 65535 * (int64_t)kC32RowsPerCta, "cg32: grid too tall");
  LXGB_REQUIRE(c32_parts(nx, ny) <= kC32MaxParts, "cg32: grid too large for the partial sums");
  LXGB_REQUIRE(work && ((uintptr_t)work & 255) == 0, "cg32: workspace must be 256-byte aligned");
  if (wbytes < lxgb_cg32_workspace_size(k)) {
    set_last_error("cg32: workspace too small");
    return LXGB_WORKSPACE_TOO_SMALL;
  }
  return LXGB_SUCCESSFUL;
}

static int* c32_codes(void* work, int k) {
  return reinterpret_cast<int*>(reinterpret_cast<char*>(work) + c32_state_bytes(k));
}

static int c32_vec_grid(int64_t n) {
  const int64_t per = (n + kC32Threads * 8 - 1) / (kC32Threads * 8);
  return (int)(per < 1 ? 1 : (per > kC32MaxParts ? kC32MaxParts : per));
}

extern "C" int lxgb_cg32_init(int32_t k, int64_t nx, int64_t ny, int64_t max_steps, void* work,
                              int64_t wbytes, void* stream) {
  int rc = c32_check(k, nx, ny, work, wbytes);
  if (rc) return rc;
  C32State s = c32_carve(work, k);
  c32_init_kernel<<<(k + 127) / 128, 128, 0, as_stream(stream)>>>(k, s, max_steps);
  return check_launch("cg32_init");
}

extern "C" int lxgb_cg32_refresh(int32_t k, int64_t nx, int64_t ny, const double* b, double* x,
                                 float* xlo, float* r, double rtol, double atol,
                                 int64_t max_steps, void* work, int64_t wbytes, void* stream) {
  int rc = c32_check(k, nx, ny, work, wbytes);
  if (rc) return rc;
  LXGB_REQUIRE(b && x && xlo && r, "cg32: null pointer");
  cudaStream_t st = as_stream(stream);
  C32State s = c32_carve(work, k);
  int* codes = c32_codes(work, k);
  dim3 g((unsigned)((ny + kC32Threads - 1) / kC32Threads),
         (unsigned)((nx + kC32RowsPerCta - 1) / kC32RowsPerCta), (unsigned)k);
  const int P = c32_parts(nx, ny);
  const bool vec = nx * ny % 4 == 0 && (((uintptr_t)x | (uintptr_t)xlo) & 15) == 0;
  const dim3 gf((unsigned)c32_vec_grid(nx * ny), (unsigned)k);
  (vec ? c32_fold_kernel<4> : c32_fold_kernel<1>)<<<gf, kC32Threads, 0, st>>>(nx * ny, s, x, xlo);
  c32_refresh_kernel<<<g, kC32Threads, 0, st>>>(nx, ny, s, b, x, r, codes, rtol, atol);
  c32_refresh_final_kernel<<<k, 32, 0, st>>>(k, s, codes, P, max_steps);
  return check_launch("cg32_refresh");
}

extern "C" int lxgb_cg32_iterate(int32_t k, int64_t nx, int64_t ny, int32_t iters, float* p,
                                 float* ap, float* xlo, float* r, void* work, int64_t wbytes,
                                 void* stream) {
  int rc = c32_check(k, nx, ny, work, wbytes);
  if (rc) return rc;
  LXGB_REQUIRE(p && ap && xlo && r, "cg32: null pointer");
  cudaStream_t st = as_stream(stream);
  C32State s = c32_carve(work, k);
  const int64_t n = nx * ny;
  dim3 gs((unsigned)((ny + kC32Threads - 1) / kC32Threads),
          (unsigned)((nx + kC32RowsPerCta - 1) / kC32RowsPerCta), (unsigned)k);
  const int Ps = c32_parts(nx, ny);
  const int Pv = c32_vec_grid(n);
  const dim3 gv((unsigned)Pv, (unsigned)k), g1((unsigned)k), bt(kC32Threads), bw(32);
  const bool vec = ny % 4 == 0 && (((uintptr_t)p | (uintptr_t)ap | (uintptr_t)xlo | (uintptr_t)r) & 15) == 0;
  float *cur = p, *nxt = ap;
  // Partials per CTA of the residual pass: sixteen where two CTAs per SM remain,
  // four where one does.  ms for 32 steps with 16, 4 and 2: 2048 x 2048, one
  // right-hand side 1.91, 1.58 and 1.67, four 4.59, 4.67 and 4.78; 701 x 1333, 64
  // 16.3, 16.7 and 17.2; 256 x 256, one 1.03, 0.73 and 0.68 (32: 2.63, 5.05, 16.7
  // and 1.49).
  int g = 16;
  if ((int64_t)k * ((Pv + g - 1) / g) < 2 * sm_count()) g = 4;
  if ((int64_t)k * ((Pv + g - 1) / g) < sm_count()) g = 2;
  auto resid = g == 16 ? c32_residual_kernel<16>
                       : (g == 4 ? c32_residual_kernel<4> : c32_residual_kernel<2>);
  const dim3 gr((unsigned)((Pv + g - 1) / g), (unsigned)k), br(kC32ResThreads);
  cudaError_t e = launch_pdl(vec ? c32_step_kernel<false, 4> : c32_step_kernel<false, 1>, gs, bt, 0,
                             st, 1, nx, ny, s, r, cur, nxt, xlo);
  for (int it = 0; it < iters && e == cudaSuccess; ++it) {
    const bool last = it + 1 == iters;
    e = launch_pdl(c32_alpha_kernel, g1, bw, 0, st, 1, k, s, Ps);
    if (e == cudaSuccess)
      e = launch_pdl(resid, gr, br, 0, st, 1, (int)n, (int)ny, Pv, s, cur, r);
    if (e == cudaSuccess) e = launch_pdl(c32_beta_kernel, g1, bw, 0, st, 1, k, s, Pv);
    if (e != cudaSuccess) break;
    if (last)
      e = launch_pdl(vec ? c32_direction_kernel<4> : c32_direction_kernel<1>, gv, bt, 0, st, 1, n, s,
                     r, cur, p, xlo);
    else
      e = launch_pdl(vec ? c32_step_kernel<true, 4> : c32_step_kernel<true, 1>, gs, bt, 0, st, 1, nx,
                     ny, s, r, cur, nxt, xlo);
    float* t = cur;
    cur = nxt;
    nxt = t;
  }
  LXGB_CUDA_TRY(e, "cg32_iterate: launch");
  return check_launch("cg32_iterate");
}

// p = r (FP32) after the first refresh.
__global__ void c32_copy_kernel(int64_t total, const float* __restrict__ src,
                                float* __restrict__ dst) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total;
       i += (int64_t)gridDim.x * blockDim.x)
    dst[i] = src[i];
}

extern "C" int lxgb_cg32_start_direction(int32_t k, int64_t n, const float* r, float* p,
                                         void* stream) {
  LXGB_REQUIRE(k >= 1 && n >= 0 && r && p, "cg32: bad arguments");
  const int64_t total = n * k;
  c32_copy_kernel<<<(unsigned)(total / 256 + 1 < 8192 ? total / 256 + 1 : 8192), 256, 0,
                    as_stream(stream)>>>(total, r, p);
  return check_launch("cg32_start_direction");
}

extern "C" int lxgb_cg32_status(int32_t k, int32_t* out, void* work, int64_t wbytes,
                                void* stream) {
  LXGB_REQUIRE(k >= 1 && out && work, "cg32: bad arguments");
  if (wbytes < lxgb_cg32_workspace_size(k)) {
    set_last_error("cg32: workspace too small");
    return LXGB_WORKSPACE_TOO_SMALL;
  }
  C32State s = c32_carve(work, k);
  c32_status_kernel<<<(k + 127) / 128, 128, 0, as_stream(stream)>>>(k, s, out);
  return check_launch("cg32_status");
}
