// General triangular solve op(T) X = B (lower/upper, trans, unit diagonal), FP64.
#include "common.cuh"
#include "trisolve.cuh"

using namespace lxgb;

extern "C" int lxgb_trsm_f64(int32_t n, int32_t nrhs, const double* t, int64_t ldt, int32_t lower,
                             int32_t trans, int32_t unit_diag, double* b, void* stream) {
  LXGB_REQUIRE(n >= 0 && nrhs >= 0, "trsm: negative size");
  if (n == 0 || nrhs == 0) return LXGB_SUCCESSFUL;
  LXGB_REQUIRE(t && b, "trsm: null pointer");
  LXGB_REQUIRE(ldt >= n, "trsm: ldt < n");
  constexpr int kMaxVectors = 65535;  // vectors per launch (grid.y)
  for (int64_t c = 0; c < nrhs; c += kMaxVectors) {
    const int k = (int)(nrhs - c < kMaxVectors ? nrhs - c : kMaxVectors);
    const int rc = trisolve_blocked(1, n, k, t, ldt, 0, lower != 0, trans != 0, unit_diag != 0,
                                    b + c * n, 0, as_stream(stream));
    if (rc) return rc;
  }
  return LXGB_SUCCESSFUL;
}
