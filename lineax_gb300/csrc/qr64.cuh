// FP64 Householder QR on thread-block clusters (qr64.cu).
#pragma once

#include "common.cuh"

namespace lxgb {

// The factorisation of h (n rows of length m, already Mᵀ) in place, with tau
// and the 32-column T blocks.  Returns 0 when launched, -1 when the shape (or
// the device) needs the general path, or a status.
int geqrf64_cluster(int64_t m, int n, double* h, double* tau, double* t, cudaStream_t st);

// op(Q) applied to nrhs vectors; the same returns.
int ormqr64_cluster(int64_t m, int n, const double* h, const double* t, int nrhs, double* c,
                    int trans, cudaStream_t st);

}  // namespace lxgb
