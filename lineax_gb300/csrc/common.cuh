// Shared helpers for the lxgb CUDA sources: status plumbing, launch checks,
// warp reductions.  Every entry point validates its arguments on the host,
// launches, and converts a launch error into LXGB_CUDA_ERROR with a message
// retrievable through lxgb_last_error().
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>
#include <stdio.h>

#include "../../include/lxgb.h"

namespace lxgb {

// Thread-local text of the last failure; defined in status.cu.
void set_last_error(const char* fmt, ...);

inline cudaStream_t as_stream(void* s) { return reinterpret_cast<cudaStream_t>(s); }

// Returns LXGB_CUDA_ERROR (and records the message) if the last launch failed.
inline int check_launch(const char* what) {
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) {
    set_last_error("%s: %s", what, cudaGetErrorString(e));
    return LXGB_CUDA_ERROR;
  }
  return LXGB_SUCCESSFUL;
}

inline int invalid(const char* fmt_msg) {
  set_last_error("%s", fmt_msg);
  return LXGB_INVALID_ARG;
}

#define LXGB_REQUIRE(cond, msg)            \
  do {                                     \
    if (!(cond)) return ::lxgb::invalid(msg); \
  } while (0)

#define LXGB_CUDA_TRY(expr, what)                                         \
  do {                                                                   \
    cudaError_t _e = (expr);                                             \
    if (_e != cudaSuccess) {                                             \
      ::lxgb::set_last_error("%s: %s", what, cudaGetErrorString(_e));    \
      return LXGB_CUDA_ERROR;                                            \
    }                                                                    \
  } while (0)

// Number of SMs of the current device (cached per process for device 0..15).
int sm_count();

// Raises kernel `fn`'s dynamic shared-memory limit to `bytes` on the current
// device.  The attribute persists in the context, so the driver is called only
// the first time a kernel needs more than it was last given (repeated driver
// calls cost microseconds of host time per launch).  Defined in status.cu.
cudaError_t ensure_dynamic_smem(const void* fn, int bytes);

// Whether a cluster of `c` CTAs of kernel `fn` (`threads` threads, `smem` bytes
// of dynamic shared memory each) can be co-scheduled on the current device; the
// kernel's limits are raised as needed.  Asked once per device and shape.
// Defined in status.cu.
bool cluster_fits(const void* fn, int c, int threads, size_t smem);

__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
__device__ __forceinline__ double warp_max(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fmax(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}

// Pivot-search key of x: |x| as its IEEE bit pattern, which orders like the
// value for every non-NaN x; NaN maps to -1 and never wins (as "|x| > v" never
// holds for NaN).  64-bit integer compares run on the integer pipe, not on
// GB300's narrow FP64 pipe.
__device__ __forceinline__ long long pivot_key(double x) {
  const long long b = __double_as_longlong(x) & 0x7FFFFFFFFFFFFFFFLL;
  return b > 0x7FF0000000000000LL ? -1LL : b;
}

// Arg-max of pivot keys with the lowest index winning ties: the combination rule
// of LAPACK idamax, which scans upward and only moves on a strictly larger
// magnitude.  Each lane first scans its own rows in increasing order with the
// same strict rule, so the warp result equals a sequential scan.
__device__ __forceinline__ void warp_argmax_first_key(long long& v, int& idx) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const long long ov = __shfl_xor_sync(0xffffffffu, v, o);
    const int oi = __shfl_xor_sync(0xffffffffu, idx, o);
    if (ov > v || (ov == v && oi < idx)) {
      v = ov;
      idx = oi;
    }
  }
}

// Programmatic dependent launch.  A kernel launched by launch_pdl may start
// while the kernel before it on the stream is still running; it must call
// pdl_wait() (all threads) before it touches anything that kernel writes, and
// may load data that no earlier kernel of the chain writes before that.
// pdl_trigger() lets the next kernel of the chain start; the next kernel's
// pdl_wait() still waits until this one has finished and its writes are
// visible, so where the trigger stands never changes a result.
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_trigger() {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

// Launch `fn` with programmatic stream serialisation (and a thread-block
// cluster of `cluster` CTAs along x when cluster > 1).
template <typename... KArgs, typename... Args>
inline cudaError_t launch_pdl(void (*fn)(KArgs...), dim3 grid, dim3 block, size_t smem,
                              cudaStream_t st, int cluster, Args... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  attr[1].id = cudaLaunchAttributeClusterDimension;
  attr[1].val.clusterDim.x = (unsigned)cluster;
  attr[1].val.clusterDim.y = 1;
  attr[1].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = cluster > 1 ? 2 : 1;
  return cudaLaunchKernelEx(&cfg, fn, static_cast<KArgs>(args)...);
}

// First maximum over a warp of (key, idx) with the lowest idx winning ties:
// three 32-bit warp reductions (REDUX) instead of a five-step 64-bit shuffle
// tree.  key 0 with idx INT_MAX marks a lane without a candidate.
__device__ __forceinline__ void warp_first_max(unsigned long long& key, int& idx) {
  const unsigned hi = (unsigned)(key >> 32), lo = (unsigned)key;
  const unsigned mh = __reduce_max_sync(0xffffffffu, hi);
  const unsigned ml = __reduce_max_sync(0xffffffffu, hi == mh ? lo : 0u);
  const unsigned mi =
      __reduce_min_sync(0xffffffffu, (hi == mh && lo == ml) ? (unsigned)idx : 0x7FFFFFFFu);
  key = ((unsigned long long)mh << 32) | ml;
  idx = (int)mi;
}

}  // namespace lxgb
