// Row interchanges x_k <-> x_{p_k}, k = 0 .. n-1, p_k >= k, as one gather, by one CTA.
//
// (P x)_i is final after interchange i, so its source is found by walking back:
// position p_i before interchange i holds what the last earlier interchange with the
// same partner put there, that is the value of a position j < i before interchange j,
// and so on.
//  * Partners: the interchanges of each partner form a linked list, built by atomics in
//    any order; a row walks its partner's list for the last interchange before its own.
//    With partners as partial pivoting of a random matrix draws them the lists have a few
//    links.  Where one has more than kSwapWalk (a companion matrix: partner n - 1 for
//    every row, n^2 / 2 links to walk) one warp orders all of them instead, 32
//    interchanges at a time.
//  * The walk back from a position by pointer jumping: a chain of n links (a cyclic
//    shift) takes log2 n rounds.
// Bound by latency.  us at n = 8192 (perm_from_swaps_kernel): random partners 16, a
// cyclic shift 16, one partner for all 36; with every row walking its list and its chain
// to the end 14, 253 and 2380; one thread running the n dependent exchanges 325.
#pragma once

#include "common.cuh"

namespace lxgb {

constexpr int kSwapWalk = 64;
enum SwapMode { kSwapShort, kSwapLong, kSwapInOrder };

// All threads of the CTA.  head and next: n entries each in shared memory; root: n more,
// shared or global.  kSwapInOrder (a partner above the diagonal: not a sequence of getrf):
// the interchanges were run one by one, in reverse order if `reverse`, and head holds
// the gather; out-of-range partners are skipped.
__device__ inline SwapMode swap_build(int n, const int32_t* p, int* head, int* next, int* root,
                                      bool reverse) {
  const int tid = threadIdx.x, nt = blockDim.x, lane = tid & 31;
  for (int i = tid; i < n; i += nt) head[i] = -1;
  __syncthreads();
  int odd = 0;
  for (int j = tid; j < n; j += nt) {
    const int q = p[j];
    if (q < j || q >= n) odd = 1;
    else if (q != j) next[j] = atomicExch(&head[q], j);
  }
  if (__syncthreads_or(odd)) {
    for (int i = tid; i < n; i += nt) head[i] = i;
    __syncthreads();
    if (tid == 0)
      for (int s = 0; s < n; ++s) {
        const int k = reverse ? n - 1 - s : s;
        const int q = p[k];
        if (q != k && q >= 0 && q < n) { const int v = head[k]; head[k] = head[q]; head[q] = v; }
      }
    __syncthreads();
    return kSwapInOrder;
  }
  // root: the latest interchange with partner k (all < k), k itself without one
  int more = 0;
  for (int k = tid; k < n; k += nt) {
    int m = -1, links = 0, j = head[k];
    for (; j >= 0 && links < kSwapWalk; j = next[j], ++links) m = max(m, j);
    if (j >= 0) more = 1;
    root[k] = m < 0 ? k : m;
  }
  const bool ordered = __syncthreads_or(more);
  if (ordered) {
    for (int i = tid; i < n; i += nt) head[i] = -1;
    __syncthreads();
    if (tid < 32) {
      constexpr int kAhead = 8;                    // groups of 32 loaded at once
      for (int b = 0; b < n; b += 32 * kAhead) {
        int q[kAhead];
#pragma unroll
        for (int u = 0; u < kAhead; ++u) q[u] = b + 32 * u + lane < n ? p[b + 32 * u + lane] : -1;
#pragma unroll
        for (int u = 0; u < kAhead; ++u) {
          const int j0 = b + 32 * u, j = j0 + lane;
          const bool in = j < n && q[u] != j;
          const unsigned same = __match_any_sync(0xffffffffu, in ? q[u] : -1 - lane);
          const unsigned before = same & ((1u << lane) - 1u);
          if (in) next[j] = before ? j0 + 31 - __clz(before) : head[q[u]];
          __syncwarp();
          if (in && (same >> lane) == 1u) head[q[u]] = j;  // the latest of the group
          __syncwarp();
        }
      }
    }
    __syncthreads();
    for (int k = tid; k < n; k += nt) root[k] = head[k] < 0 ? k : head[k];
    __syncthreads();
  }
  int moved;
  do {                                             // every entry moves towards its chain's end
    moved = 0;
    for (int k = tid; k < n; k += nt) {
      const int a = root[k], b = root[a];
      if (a != b) {
        root[k] = root[b];
        moved = 1;
      }
    }
  } while (__syncthreads_or(moved));
  return ordered ? kSwapLong : kSwapShort;
}

// Where (P x)_i comes from (kSwapInOrder: in the order run).
__device__ inline int swap_source(SwapMode mode, int i, const int32_t* p, const int* head,
                                  const int* next, const int* root) {
  if (mode == kSwapInOrder) return head[i];
  const int q = p[i];
  if (q == i) return root[i];
  int from = -1;
  if (mode == kSwapLong) {
    from = next[i];
  } else {
    for (int j = head[q]; j >= 0; j = next[j])
      if (j < i) from = max(from, j);
  }
  return from < 0 ? q : root[from];
}

}  // namespace lxgb
