// kclpp_extract.cu -- see kclpp_extract.cuh.
//
// The order is a stable radix sort by 8-bit digits, least significant first,
// over the digits the largest key has: per digit a count of each tile's
// digits, a scan of the counts (digit-major, so that tiles keep their order
// within a digit) and a scatter.  What bounds it at the sizes of a report
// (10^4 .. 10^6 vertices, 3 or 4 digits) is launches.  A run of 16 passes with
// five reports on 60,000 vertices took 14.8 ms with the order and the prefix
// scan on the host, 6.0 with them here.
#include <algorithm>

#include "kclpp_dev.cuh"
#include "kclpp_extract.cuh"

namespace kclpp {

namespace {

constexpr int kThreads = 256;
constexpr int kWarps = kThreads / 32;
constexpr int kPer = 8;                      // keys per thread
constexpr uint32_t kTile = kThreads * kPer;  // 2048
inline uint32_t tiles_of(uint32_t n) { return (n + kTile - 1) / kTile; }

// Descending order: a larger key has the smaller digit.
__device__ __forceinline__ uint32_t digit_of(unsigned long long key, int shift) {
  return 255u - (uint32_t)((key >> shift) & 255u);
}

// hist[digit * tiles + tile] = keys of the tile with that digit.
__global__ void __launch_bounds__(kThreads) k_digits(const unsigned long long *keys, uint32_t n, int shift,
                                                     uint32_t tiles, uint32_t *hist) {
  __shared__ uint32_t cnt[256];
  cnt[threadIdx.x] = 0;
  __syncthreads();
  const uint32_t base = blockIdx.x * kTile;
#pragma unroll
  for (int q = 0; q < kPer; ++q) {
    const uint32_t i = base + q * kThreads + threadIdx.x;
    if (i < n) atomicAdd(&cnt[digit_of(keys[i], shift)], 1u);
  }
  __syncthreads();
  hist[threadIdx.x * tiles + blockIdx.x] = cnt[threadIdx.x];
}

// Exclusive scan of v[0, m) in place, one block.
__global__ void __launch_bounds__(1024) k_scan(uint32_t *v, uint32_t m) {
  __shared__ uint32_t part[32];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  uint32_t carry = 0;
  for (uint32_t b = 0; b < m; b += 4096) {
    uint32_t x[4], sum = 0;
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const uint32_t i = b + threadIdx.x * 4 + q;
      x[q] = i < m ? v[i] : 0u;
      sum += x[q];
    }
    uint32_t inc = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t y = __shfl_up_sync(KCL_FULL, inc, o);
      if (lane >= o) inc += y;
    }
    if (lane == 31) part[wid] = inc;
    __syncthreads();
    uint32_t p = part[lane];
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t y = __shfl_up_sync(KCL_FULL, p, o);
      if (lane >= o) p += y;
    }
    const uint32_t before = wid ? __shfl_sync(KCL_FULL, p, wid - 1) : 0u;
    const uint32_t all = __shfl_sync(KCL_FULL, p, 31);
    uint32_t at = carry + before + inc - sum;
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const uint32_t i = b + threadIdx.x * 4 + q;
      if (i < m) v[i] = at;
      at += x[q];
    }
    carry += all;
    __syncthreads();  // part is reused
  }
}

// Each key to its place: a warp owns 256 consecutive keys of the tile and
// ranks them 32 at a time, so equal digits keep their order.  ids == nullptr:
// the ids are the positions (first digit).
__global__ void __launch_bounds__(kThreads) k_place(const unsigned long long *keys, const uint32_t *ids, uint32_t n,
                                                    int shift, uint32_t tiles, const uint32_t *hist,
                                                    unsigned long long *keys_out, uint32_t *ids_out) {
  __shared__ uint32_t cnt[kWarps][256];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  for (int i = lane; i < 256; i += 32) cnt[wid][i] = 0;
  __syncwarp();
  const uint32_t base = blockIdx.x * kTile + wid * 32 * kPer + lane;
  unsigned long long key[kPer];
  uint32_t rank[kPer];
#pragma unroll
  for (int q = 0; q < kPer; ++q) {
    const uint32_t i = base + 32 * q;
    const bool live = i < n;
    key[q] = live ? keys[i] : 0ull;
    const uint32_t d = live ? digit_of(key[q], shift) : 256u;
    const uint32_t same = __match_any_sync(KCL_FULL, d);
    const uint32_t before = (uint32_t)__popc(same & dev::lanemask_lt());
    uint32_t at = 0;
    if (live) at = cnt[wid][d];
    __syncwarp();
    if (live && before == 0) cnt[wid][d] = at + (uint32_t)__popc(same);
    __syncwarp();
    rank[q] = at + before;
  }
  __syncthreads();
  {  // per digit: where each warp's keys of it start
    uint32_t at = hist[threadIdx.x * tiles + blockIdx.x];
#pragma unroll
    for (int w = 0; w < kWarps; ++w) {
      const uint32_t c = cnt[w][threadIdx.x];
      cnt[w][threadIdx.x] = at;
      at += c;
    }
  }
  __syncthreads();
#pragma unroll
  for (int q = 0; q < kPer; ++q) {
    const uint32_t i = base + 32 * q;
    if (i >= n) continue;
    const uint32_t to = cnt[wid][digit_of(key[q], shift)] + rank[q];
    keys_out[to] = key[q];
    ids_out[to] = ids ? ids[i] : i;
  }
}

__global__ void k_levels(const uint32_t *ids, uint32_t n, uint32_t *order, uint32_t *level) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const uint32_t v = ids ? ids[i] : i;
  if (order != ids) order[i] = v;
  level[v] = i;
}

__global__ void k_widen(const uint32_t *a, uint32_t n, unsigned long long *b) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) b[i] = a[i];
}

// ---- densest prefix ---------------------------------------------------------
template <typename T>
__device__ __forceinline__ T block_sum(T x, T *part) {
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  x = dev::warp_sum(x);
  __syncthreads();
  if (lane == 0) part[wid] = x;
  __syncthreads();
  T y = 0;
#pragma unroll
  for (int w = 0; w < kWarps; ++w) y += part[w];
  return y;
}

template <typename C>
__global__ void __launch_bounds__(kThreads) k_tile_sums(const C *cnt, uint32_t n, unsigned long long *sums) {
  __shared__ unsigned long long part[kWarps];
  unsigned long long s = 0;
#pragma unroll
  for (int q = 0; q < kPer; ++q) {
    const uint32_t i = blockIdx.x * kTile + q * kThreads + threadIdx.x;
    if (i < n) s += cnt[i];
  }
  s = block_sum(s, part);
  if (threadIdx.x == 0) sums[blockIdx.x] = s;
}

struct Cand {
  double dens;
  unsigned long long sum;
  uint32_t i;
};
// The scan keeps the first strictly larger density: larger, then earlier.
__device__ __forceinline__ bool better(double d, uint32_t i, double e, uint32_t j) { return d > e || (d == e && i < j); }
__device__ __forceinline__ Cand warp_best(Cand c) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const double d = __shfl_xor_sync(KCL_FULL, c.dens, o);
    const unsigned long long s = __shfl_xor_sync(KCL_FULL, c.sum, o);
    const uint32_t i = __shfl_xor_sync(KCL_FULL, c.i, o);
    if (better(d, i, c.dens, c.i)) c = {d, s, i};
  }
  return c;
}

// Best prefix that ends in each tile; the tile's start sum from the sums of
// the tiles before it.
template <typename C>
__global__ void __launch_bounds__(kThreads) k_tile_best(const C *cnt, uint32_t n, const unsigned long long *sums,
                                                        Cand *cand) {
  __shared__ unsigned long long part[kWarps], wsum[kWarps];
  __shared__ Cand wbest[kWarps];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  unsigned long long before = 0;
  for (uint32_t t = threadIdx.x; t < blockIdx.x; t += kThreads) before += sums[t];
  before = block_sum(before, part);
  const uint32_t base = blockIdx.x * kTile + threadIdx.x * kPer;
  unsigned long long x[kPer], own = 0;
#pragma unroll
  for (int q = 0; q < kPer; ++q) {
    x[q] = base + q < n ? cnt[base + q] : 0;
    own += x[q];
  }
  unsigned long long inc = own;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const unsigned long long y = __shfl_up_sync(KCL_FULL, inc, o);
    if (lane >= o) inc += y;
  }
  if (lane == 31) wsum[wid] = inc;
  __syncthreads();
  unsigned long long at = before + inc - own;
  for (int w = 0; w < wid; ++w) at += wsum[w];
  Cand c{-1.0, 0, 0xffffffffu};
#pragma unroll
  for (int q = 0; q < kPer; ++q) {
    const uint32_t i = base + q;
    if (i < n) {
      at += x[q];
      const double d = __ddiv_rn(__ull2double_rn(at), (double)(i + 1));
      if (d > c.dens) c = {d, at, i};
    }
  }
  c = warp_best(c);
  if (lane == 0) wbest[wid] = c;
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int w = 1; w < kWarps; ++w)
      if (better(wbest[w].dens, wbest[w].i, c.dens, c.i)) c = wbest[w];
    cand[blockIdx.x] = c;
  }
}

__global__ void __launch_bounds__(32) k_best(const Cand *cand, const unsigned long long *sums, uint32_t tiles,
                                             PrefixBest *best) {
  Cand c{-1.0, 0, 0xffffffffu};
  unsigned long long total = 0;
  for (uint32_t t = threadIdx.x; t < tiles; t += 32) {
    total += sums[t];
    if (better(cand[t].dens, cand[t].i, c.dens, c.i)) c = cand[t];
  }
  c = warp_best(c);
  total = dev::warp_sum(total);
  if (threadIdx.x == 0) *best = {c.dens, c.sum, total, 0, c.i + 1};
}

template <typename C>
cudaError_t densest(const C *cnt, uint32_t n, OrderScratch &s, PrefixBest *best, cudaStream_t st, uint64_t *launches) {
  const uint32_t tiles = tiles_of(n);
  unsigned long long *sums = s.sums;
  Cand *cand = reinterpret_cast<Cand *>(s.sums + tiles);
  k_tile_sums<C><<<tiles, kThreads, 0, st>>>(cnt, n, sums);
  k_tile_best<C><<<tiles, kThreads, 0, st>>>(cnt, n, sums, cand);
  k_best<<<1, 32, 0, st>>>(cand, sums, tiles, best);
  *launches += 3;
  return cudaGetLastError();
}

}  // namespace

cudaError_t order_scratch_make(OrderScratch &s, uint32_t n) {
  if (s.keys && s.n >= n) return cudaSuccess;
  order_scratch_free(s);
  const size_t m = std::max<uint32_t>(n, 1), t = tiles_of((uint32_t)m);
  cudaError_t e = cudaMalloc((void **)&s.keys, m * 8);
  if (e == cudaSuccess) e = cudaMalloc((void **)&s.ids, m * 4);
  if (e == cudaSuccess) e = cudaMalloc((void **)&s.hist, t * 256 * 4);
  if (e == cudaSuccess) e = cudaMalloc((void **)&s.sums, t * 8 + t * sizeof(Cand));
  if (e != cudaSuccess) order_scratch_free(s);
  else s.n = n;
  return e;
}

void order_scratch_free(OrderScratch &s) {
  cudaFree(s.keys); cudaFree(s.ids); cudaFree(s.hist); cudaFree(s.sums);
  s = OrderScratch{};
}

cudaError_t order_by_key(unsigned long long *keys, uint32_t n, uint64_t key_max, OrderScratch &s, uint32_t *order,
                         uint32_t *level, cudaStream_t st, uint64_t *launches) {
  if (!n) return cudaSuccess;
  const uint32_t tiles = tiles_of(n);
  int digits = 0;
  while (digits < 8 && (key_max >> (8 * digits))) ++digits;
  unsigned long long *kin = keys, *kout = s.keys;
  const uint32_t *iin = nullptr;
  // the last digit writes `order`: alternate backwards from it
  for (int d = 0; d < digits; ++d) {
    uint32_t *iout = ((digits - 1 - d) & 1) ? s.ids : order;
    k_digits<<<tiles, kThreads, 0, st>>>(kin, n, 8 * d, tiles, s.hist);
    k_scan<<<1, 1024, 0, st>>>(s.hist, 256 * tiles);
    k_place<<<tiles, kThreads, 0, st>>>(kin, iin, n, 8 * d, tiles, s.hist, kout, iout);
    std::swap(kin, kout);
    iin = iout;
    *launches += 3;
  }
  k_levels<<<(n + 255) / 256, 256, 0, st>>>(iin, n, order, level);
  *launches += 1;
  return cudaGetLastError();
}

cudaError_t order_by_key32(const uint32_t *keys, uint32_t n, uint32_t key_max, OrderScratch &s,
                           unsigned long long *tmp, uint32_t *order, uint32_t *level, cudaStream_t st,
                           uint64_t *launches) {
  if (!n) return cudaSuccess;
  k_widen<<<(n + 255) / 256, 256, 0, st>>>(keys, n, tmp);
  *launches += 1;
  return order_by_key(tmp, n, key_max, s, order, level, st, launches);
}

cudaError_t densest_prefix(const unsigned long long *cnt, uint32_t n, OrderScratch &s, PrefixBest *best,
                           cudaStream_t st, uint64_t *launches) {
  return densest(cnt, n, s, best, st, launches);
}
cudaError_t densest_prefix32(const uint32_t *cnt, uint32_t n, OrderScratch &s, PrefixBest *best, cudaStream_t st,
                             uint64_t *launches) {
  return densest(cnt, n, s, best, st, launches);
}

}  // namespace kclpp
