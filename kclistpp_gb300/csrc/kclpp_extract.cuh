// kclpp_extract.cuh -- device side of the reports: the order of the vertices
// by decreasing load and the densest prefix of a per-position clique count
// (CDF_NodeCmp + qsort and the scan of kCDensestNoAtom.c:322-349).
#pragma once

#include <cstddef>
#include <cstdint>
#include <cuda_runtime.h>

#include "kclpp_internal.h"

namespace kclpp {

// Scratch of the order: a second key and id array and the digit counts, kept
// with the graph or sample that is reported on.
struct OrderScratch {
  unsigned long long *keys = nullptr;  // n
  uint32_t *ids = nullptr;             // n
  uint32_t *hist = nullptr;
  unsigned long long *sums = nullptr;
  uint32_t n = 0;
};
cudaError_t order_scratch_make(OrderScratch &s, uint32_t n);
void order_scratch_free(OrderScratch &s);

// Vertices by decreasing keys[v], ties by ascending v: order[i] and
// level[order[i]] = i.  keys (n) is overwritten; key_max bounds every key.
// Enqueues on st; *launches grows by the kernels launched.
cudaError_t order_by_key(unsigned long long *keys, uint32_t n, uint64_t key_max, OrderScratch &s, uint32_t *order,
                         uint32_t *level, cudaStream_t st, uint64_t *launches);
// The same from 32-bit keys (left as they are; widened into s's arrays).
cudaError_t order_by_key32(const uint32_t *keys, uint32_t n, uint32_t key_max, OrderScratch &s,
                           unsigned long long *tmp, uint32_t *order, uint32_t *level, cudaStream_t st,
                           uint64_t *launches);

// First strictly largest prefix density of cnt[0..n): the prefix's length and
// sum, the sum of all of cnt, as the reference's scan finds them.  edges starts
// at 0, for the caller to count the edges inside the prefix.
struct PrefixBest {
  double density;
  unsigned long long cliques, total, edges;
  uint32_t n;
};
cudaError_t densest_prefix(const unsigned long long *cnt, uint32_t n, OrderScratch &s, PrefixBest *best,
                           cudaStream_t st, uint64_t *launches);
cudaError_t densest_prefix32(const uint32_t *cnt, uint32_t n, OrderScratch &s, PrefixBest *best, cudaStream_t st,
                             uint64_t *launches);

}  // namespace kclpp
