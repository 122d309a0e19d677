// Multi-CTA triangular solve shared by trsm (trsm.cu) and getrs (lu.cu).
#pragma once

#include "common.cuh"

namespace lxgb {

constexpr int kTsNB = 64;  // unknowns per step

// op(T) x = b in place for `nrhs` vectors (vector c at x + c * n) of each of
// `batch` systems (strides stride_t, stride_x), T row-major with leading
// dimension ldt: in one launch for few vectors and for many, else one per kTsNB
// unknowns.  nrhs and batch at most 65535.
int trisolve_blocked(int64_t batch, int n, int nrhs, const double* t, int64_t ldt,
                     int64_t stride_t, int lower, int trans, int unit, double* x,
                     int64_t stride_x, cudaStream_t st);

}  // namespace lxgb
