// kclpp_sample.cu -- Seq-Sampling++ on the GPU (kCDensestSamplingKclistpp.c):
// the clique sample kept in device memory, the "++" passes over it, and the
// report (densest prefix of the sampled loads, exact count inside it, bound).
//
// Sampling kernel: one CTA per root vertex s (persistent CTAs, roots by
// decreasing out-degree from an atomic counter).  The CTA loads N+(s) and the
// members' keys and builds G_s as bitmap rows (row i = the members of N+(s)
// that are out-neighbours of the i-th one) in shared memory; its warps take the
// root edges (s, t) and walk each edge's clique tree, a word of the candidate
// set per lane, down to the last two levels, where a lane stands for a last
// member v and runs through the members u before it whose row holds v.  A
// clique is kept when its key sum passes the threshold (kclpp_sample.cuh); kept
// rows are appended at an atomic cursor.  Instruction issue bounds it (~20
// instructions of hashing per clique): a lane per clique keeps the lanes busy,
// where a thread per root edge diverged (4.9 ms for the 2.1e8 4-cliques of an
// RMAT-16 graph).  Roots beyond out-degree 1024 (more than 32 words a row) take
// the thread-per-edge kernel, rows in a per-CTA global slab.  The order of the
// rows is arbitrary; they are then grouped by wave, and nothing downstream
// depends on the order inside a wave.
//
// "++" pass: W waves (a fixed byte per kept clique).  Wave w: every clique of
// the wave adds one to its argmin (values as the earlier waves left them).
// Integer adds commute, so the result is the same for every schedule.  A
// wave's rows lie together, and one launch runs it: a vertex's value is a pair
// (load, increments of the wave before), the launch folds each pair into the
// next buffer while its cliques add to that buffer's increments.  Two launches
// a wave over the whole sample's wave bytes took 19 us where this takes ~3.
#include <algorithm>
#include <cmath>
#include <cstring>
#include <memory>
#include <numeric>
#include <vector>

#include <cuda_runtime.h>

#include "kclpp_extract.cuh"
#include "kclpp_internal.h"
#include "kclpp_kernels.cuh"
#include "kclpp_sample.cuh"

using namespace kclpp;

#define SCUDA(call)                                                                           \
  do {                                                                                        \
    cudaError_t e_ = (call);                                                                  \
    if (e_ != cudaSuccess)                                                                    \
      return set_error(e_ == cudaErrorMemoryAllocation ? KCLPP_ERR_NOMEM : KCLPP_ERR_CUDA,    \
                       "%s: %s", #call, cudaGetErrorString(e_));                               \
  } while (0)

#define STRY(call)                         \
  do {                                     \
    kclpp_status s_ = (call);              \
    if (s_ != KCLPP_OK) return s_;         \
  } while (0)

namespace {

constexpr int kSampleThreads = 512;
constexpr uint32_t kWarpRoots = 1024;  // out-degree bound of the warp-per-edge kernel
// Out-degree bounds and CTA widths of its launch groups: small roots have few
// edges to share out and little shared memory to hold, so many narrow CTAs.
// (Bounds 128 and 48 with 1024 threads for the largest: no difference.)
constexpr uint32_t kGroupDeg[3] = {256, 64, 0};
constexpr int kGroupThreads[3] = {512, 256, 128};
constexpr int kPassThreads = 256;

struct SampleArgs {
  const uint64_t *off;
  const uint32_t *cols;
  const uint32_t *roots;  // this group's roots
  uint32_t num_roots;
  uint32_t dmax;          // largest out-degree in the group
  uint32_t ws;            // words per bitmap row
  uint32_t *work;         // root counter (zeroed)
  uint32_t *slab;         // thread-per-edge kernel: rows in global memory
  uint64_t slab_words;    // per CTA
  uint64_t seed, threshold;
  int all;
  uint32_t waves;
  uint32_t *rows;         // kept cliques, K ids each
  uint8_t *wave;
  unsigned long long cap;
  unsigned long long *count;
  unsigned long long *wave_at;  // next free row of each wave, or nullptr: rows in any order, counted in count
  const uint4 *bit_rows;  // the graph's bitmap rows (dev::PassArgs)
  const uint32_t *bits;
};

template <int K>
struct DevEmit {
  const uint32_t *list;
  uint32_t s;
  uint32_t *rows;
  uint8_t *wave;
  unsigned long long cap;
  unsigned long long *count, *wave_at;
  uint64_t threshold;
  bool all;
  uint32_t waves;
  __device__ __forceinline__ void operator()(uint64_t h, const uint32_t *path, uint32_t v) const {
    if (!smp::kept(h, threshold, all)) return;
    const uint32_t w = smp::wave_of(h, waves);
    const unsigned long long pos = atomicAdd(wave_at ? wave_at + w : count, 1ull);
    if (pos >= cap) return;  // counted only: the host grows the buffer and samples again
    smp::write_row<K>(rows + pos * K, list, s, path, v);
    wave[pos] = (uint8_t)w;
  }
};

// Shared memory: keys (dmax u64), list (dmax u32); the rows are in the slab.
template <int K>
__global__ void __launch_bounds__(kSampleThreads) k_sample(SampleArgs a) {
  extern __shared__ __align__(16) unsigned char smem[];
  uint64_t *keys = reinterpret_cast<uint64_t *>(smem);
  uint32_t *list = reinterpret_cast<uint32_t *>(keys + a.dmax);
  uint32_t *rows = a.slab + (size_t)blockIdx.x * a.slab_words;
  __shared__ uint32_t s_root, s_edge;
  for (;;) {
    if (threadIdx.x == 0) {
      s_root = atomicAdd(a.work, 1u);
      s_edge = 0;
    }
    __syncthreads();
    const uint32_t ri = s_root;
    if (ri >= a.num_roots) break;
    const uint32_t s = a.roots[ri];
    const uint64_t o = a.off[s];
    const uint32_t d = (uint32_t)(a.off[s + 1] - o);  // K - 1 <= d <= dmax (host)
    for (uint32_t i = threadIdx.x; i < d; i += blockDim.x) {
      const uint32_t x = a.cols[o + i];
      list[i] = x;
      keys[i] = smp::vertex_key(a.seed, x);
    }
    __syncthreads();
    for (uint32_t i = threadIdx.x; i < d; i += blockDim.x)
      smp::build_row(i, list, a.off, a.cols, rows + (size_t)i * a.ws);
    __syncthreads();
    DevEmit<K> em{list, s, a.rows, a.wave, a.cap, a.count, a.wave_at, a.threshold, a.all != 0, a.waves};
    const uint64_t hs = smp::vertex_key(a.seed, s);
    for (;;) {
      const uint32_t t = atomicAdd(&s_edge, 1u);
      if (t >= d) break;
      if (t + 2 < (uint32_t)K) continue;  // row t holds fewer than K - 2 candidates
      smp::edge_cliques<K>(t, hs, rows, a.ws, keys, em);
    }
    __syncthreads();  // the next root overwrites list, keys, rows and s_root
  }
}

// Shared memory of a warp-per-edge CTA: keys, list, position table, rows, then
// per warp the candidates' words, a group's row offsets and key sums, and the
// candidates' local ids.
struct WarpLayout {
  size_t list, tab, rows, warp, warp_bytes, total;
};
__host__ __device__ inline WarpLayout warp_layout(uint32_t dmax, int nw) {
  WarpLayout L;
  size_t at = (size_t)dmax * 8;
  L.list = at; at = dev::align16(at + (size_t)dmax * 4);
  L.tab = at; at = dev::align16(at + ((size_t)4 << dev::tab_bits(dmax)));
  L.rows = at; at = dev::align16(at + (size_t)dev::tri_off(dmax) * 4);
  L.warp = at;
  L.warp_bytes = dev::align16(32 * 4 + 32 * 8 + (size_t)dmax * 2);
  L.total = at + nw * L.warp_bytes + 128;  // a column read may start in the last row and end 31 words on
  return L;
}

template <int K>
struct WarpWalk {
  const SampleArgs &a;
  const uint32_t *rows, *list;
  const uint64_t *keys;
  uint32_t *ro;    // 32
  uint64_t *hk;    // 32
  uint16_t *mem;   // dmax
  uint32_t s;
  int lane;
  uint32_t path[K];  // local ids after the root, largest first

  // A kept clique (path[0 .. K - 3], then u, v): appended by the lanes that are here.
  __device__ __forceinline__ void emit(uint64_t h, uint32_t u, uint32_t v) {
    if (!smp::kept(h, a.threshold, a.all != 0)) return;
    unsigned long long pos = 0;
    if (a.wave_at) {
      pos = atomicAdd(a.wave_at + smp::wave_of(h, a.waves), 1ull);
    } else {
      const uint32_t here = __activemask();
      const int first = __ffs((int)here) - 1;
      if (lane == first) pos = atomicAdd(a.count, (unsigned long long)__popc(here));
      pos = __shfl_sync(here, pos, first) + (uint32_t)__popc(here & dev::lanemask_lt());
    }
    if (pos >= a.cap) return;  // counted only: the host grows the buffer and samples again
    uint32_t *row = a.rows + pos * K;
    row[0] = list[v];
    row[1] = list[K == 3 ? path[0] : u];
#pragma unroll
    for (int i = 2; i <= K - 2; ++i) row[i] = list[path[K - 2 - i]];
    row[K - 1] = s;
    a.wave[pos] = (uint8_t)smp::wave_of(h, a.waves);
  }

  // The last two levels over P: a lane per last member v, which runs through
  // the u of 32 rows that hold it.
  __device__ __forceinline__ void pairs(uint32_t P, uint64_t h) {
    __syncwarp();
    const int np = dev::list_members(P, mem, lane);
    __syncwarp();
    for (int g0 = 0; g0 < np; g0 += 32) {
      const int ng = np - g0 < 32 ? np - g0 : 32;
      uint32_t off = 0;
      if (lane < ng) {
        const uint32_t u = mem[g0 + lane];
        off = dev::tri_off(u);
        hk[lane] = h + keys[u];
      }
      ro[lane] = off;
      __syncwarp();
      for (int i0 = 0; i0 < g0 + ng; i0 += 32) {
        const int i = i0 + lane;
        if (i < np) {
          const uint32_t v = mem[i];
          const uint64_t kv = keys[v];
          uint32_t T = dev::column_bits(rows, ro, v, i, g0, ng);
          while (T) {
            const int g = __ffs((int)T) - 1;
            T &= T - 1;
            emit(hk[g] + kv, mem[g0 + g], v);
          }
        }
      }
      __syncwarp();
    }
  }

  template <int L>
  __device__ __forceinline__ void walk(uint32_t P, uint64_t h) {
    if constexpr (L == 2) {
      pairs(P, h);
    } else if constexpr (L == 1) {
      uint32_t nz = __ballot_sync(KCL_FULL, P != 0);
      while (nz) {
        const int w = __ffs((int)nz) - 1;
        nz &= nz - 1;
        const uint32_t word = __shfl_sync(KCL_FULL, P, w);
        if ((word >> lane) & 1u) {
          const uint32_t v = ((uint32_t)w << 5) | (uint32_t)lane;
          emit(h + keys[v], 0u, v);
        }
        __syncwarp();
      }
    } else {
      uint32_t nz = __ballot_sync(KCL_FULL, P != 0);
      while (nz) {
        const int w = __ffs((int)nz) - 1;
        nz &= nz - 1;
        uint32_t word = __shfl_sync(KCL_FULL, P, w);
        while (word) {
          const uint32_t u = ((uint32_t)w << 5) | (uint32_t)(__ffs((int)word) - 1);
          word &= word - 1;
          const uint32_t Q = lane <= w ? P & rows[dev::tri_off(u) + lane] : 0u;
          if (__reduce_add_sync(KCL_FULL, (uint32_t)__popc(Q)) < (uint32_t)(L - 1)) continue;
          path[K - 1 - L] = u;
          walk<L - 1>(Q, h + keys[u]);
        }
      }
    }
  }
};

template <int K>
__global__ void __launch_bounds__(kGroupThreads[0]) k_sample_warps(SampleArgs a) {
  extern __shared__ __align__(16) unsigned char smem[];
  const int nw = (int)(blockDim.x >> 5), tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  const WarpLayout lay = warp_layout(a.dmax, nw);
  uint64_t *keys = reinterpret_cast<uint64_t *>(smem);
  uint32_t *list = reinterpret_cast<uint32_t *>(smem + lay.list);
  uint32_t *tab = reinterpret_cast<uint32_t *>(smem + lay.tab);
  uint32_t *rows = reinterpret_cast<uint32_t *>(smem + lay.rows);
  unsigned char *mine = smem + lay.warp + (size_t)wid * lay.warp_bytes;
  __shared__ uint32_t s_root, s_edge;
  dev::PassArgs g{};
  g.off = a.off;
  g.cols = a.cols;
  g.bit_rows = a.bit_rows;
  g.bits = a.bits;
  for (;;) {
    if (tid == 0) {
      s_root = atomicAdd(a.work, 1u);
      s_edge = 0;
    }
    __syncthreads();
    const uint32_t ri = s_root;
    if (ri >= a.num_roots) break;
    const uint32_t s = a.roots[ri];
    const uint64_t o = a.off[s];
    const int d = (int)(a.off[s + 1] - o);  // K - 1 <= d <= dmax (host)
    const int tb = dev::tab_bits((uint32_t)d);
    for (int i = tid; i < d; i += blockDim.x) {
      const uint32_t x = a.cols[o + i];
      list[i] = x;
      keys[i] = smp::vertex_key(a.seed, x);
    }
    for (int i = tid; i < (int)dev::tri_off((uint32_t)d); i += blockDim.x) rows[i] = 0;
    for (int i = tid; i < 1 << tb; i += blockDim.x) tab[i] = dev::kTabEmpty;
    __syncthreads();
    for (int i = tid; i < d; i += blockDim.x) dev::tab_insert(tab, tb, list[i], i);
    __syncthreads();
    dev::induce_rows(
        g, list, d, tab, tb, wid, nw, lane,
        [&](int i, int w, bool hit) {
          const uint32_t m = __ballot_sync(KCL_FULL, hit);
          if (lane == 0) rows[dev::tri_off((uint32_t)i) + w] = m;
        },
        [&](int i, int j) { atomicOr(&rows[dev::tri_off((uint32_t)i) + (j >> 5)], 1u << (j & 31)); });
    __syncthreads();
    WarpWalk<K> wk{a, rows, list, keys, reinterpret_cast<uint32_t *>(mine), reinterpret_cast<uint64_t *>(mine + 128),
                   reinterpret_cast<uint16_t *>(mine + 384), s, lane, {}};
    const uint64_t hs = smp::vertex_key(a.seed, s);
    for (;;) {
      int t = 0;
      if (lane == 0) t = d - 1 - (int)atomicAdd(&s_edge, 1u);  // the largest candidate sets first
      t = __shfl_sync(KCL_FULL, t, 0);
      if (t < K - 2) break;  // row t holds fewer than K - 2 candidates
      wk.path[0] = (uint32_t)t;
      wk.template walk<K - 2>(lane <= (t >> 5) ? rows[dev::tri_off((uint32_t)t) + lane] : 0u, hs + keys[t]);
      __syncwarp();
    }
    __syncthreads();  // the next root overwrites list, keys, rows and s_root
  }
}

// The sample grouped by wave: the rows of each wave are counted (cnt[w + 1]),
// and moved to the wave's range (cur[w]: its next free row).
__global__ void __launch_bounds__(256) k_wave_count(const uint8_t *wave, uint64_t n_rows, unsigned long long *cnt) {
  __shared__ uint32_t c[smp::kMaxWaves];
  c[threadIdx.x] = 0;
  __syncthreads();
  const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
  for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n_rows; i += stride) atomicAdd(&c[wave[i]], 1u);
  __syncthreads();
  if (c[threadIdx.x]) atomicAdd(&cnt[threadIdx.x + 1], (unsigned long long)c[threadIdx.x]);
}
// A block's tile of rows at a time: places inside a wave by shared counters,
// one global add per wave and tile.
__global__ void __launch_bounds__(256) k_wave_move(const uint32_t *rows, const uint8_t *wave, uint64_t n_rows, int k,
                                                   unsigned long long *cur, uint32_t *rows_out, uint8_t *wave_out) {
  constexpr int kPer = 8;
  __shared__ uint32_t c[smp::kMaxWaves];
  __shared__ unsigned long long at[smp::kMaxWaves];
  const uint64_t tile = (uint64_t)blockDim.x * kPer;
  for (uint64_t b = blockIdx.x * tile; b < n_rows; b += gridDim.x * tile) {
    c[threadIdx.x] = 0;
    __syncthreads();
    uint32_t place[kPer], w[kPer];
#pragma unroll
    for (int q = 0; q < kPer; ++q) {
      const uint64_t i = b + q * blockDim.x + threadIdx.x;
      w[q] = i < n_rows ? wave[i] : smp::kMaxWaves;
      place[q] = i < n_rows ? atomicAdd(&c[w[q]], 1u) : 0u;
    }
    __syncthreads();
    if (c[threadIdx.x]) at[threadIdx.x] = atomicAdd(&cur[threadIdx.x], (unsigned long long)c[threadIdx.x]);
    __syncthreads();
#pragma unroll
    for (int q = 0; q < kPer; ++q) {
      const uint64_t i = b + q * blockDim.x + threadIdx.x;
      if (i >= n_rows) continue;
      const uint64_t to = at[w[q]] + place[q];
      for (int j = 0; j < k; ++j) rows_out[to * k + j] = rows[i * k + j];
      wave_out[to] = (uint8_t)w[q];
    }
    __syncthreads();
  }
}

// A vertex's value in the passes: x its load before the previous wave, y that
// wave's increments.
__global__ void k_open(uint32_t n, const uint32_t *rho, uint2 *b0, uint2 *b1, uint2 *b2) {
  const uint32_t v = blockIdx.x * blockDim.x + threadIdx.x;
  if (v >= n) return;
  b0[v] = make_uint2(rho[v], 0u);
  b1[v] = make_uint2(0u, 0u);
  b2[v] = make_uint2(0u, 0u);
}
__global__ void k_close(uint32_t n, const uint2 *b, uint32_t *rho) {
  const uint32_t v = blockIdx.x * blockDim.x + threadIdx.x;
  if (v < n) rho[v] = b[v].x + b[v].y;
}
// One wave, rows [lo, hi): in holds the values, out receives their fold and the
// cliques' units (its increments are zero at the start), clear's increments are
// zeroed for the wave after.
template <int K>
__global__ void __launch_bounds__(kPassThreads) k_wave(const uint32_t *rows, uint64_t lo, uint64_t hi, uint32_t n,
                                                       const uint2 *in, uint2 *out, uint2 *clear) {
  const uint64_t stride = (uint64_t)gridDim.x * blockDim.x, first = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
  for (uint64_t i = lo + first; i < hi; i += stride) {
    uint32_t m[K];
    if constexpr (K == 4) {
      const uint4 r = __ldg(reinterpret_cast<const uint4 *>(rows) + i);
      m[0] = r.x; m[1] = r.y; m[2] = r.z; m[3] = r.w;
    } else {
#pragma unroll
      for (int j = 0; j < K; ++j) m[j] = __ldg(rows + i * K + j);
    }
    // smallest value, ties to the earliest member (smp::argmin_member)
    uint32_t g = m[0], gv = 0xffffffffu;
#pragma unroll
    for (int j = 0; j < K; ++j) {
      const uint2 x = in[m[j]];
      const uint32_t v = x.x + x.y;
      if (j == 0 || v < gv) {
        g = m[j];
        gv = v;
      }
    }
    atomicAdd(&out[g].y, 1u);
  }
  for (uint64_t v = first; v < n; v += stride) {
    const uint2 x = in[v];
    out[v].x = x.x + x.y;
    clear[v].y = 0;
  }
}

__global__ void k_push(const uint32_t *rows, uint64_t n_rows, int k, const uint32_t *rank, uint32_t *push) {
  const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
  for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n_rows; i += stride)
    atomicAdd(&push[smp::max_rank(rows + i * (uint64_t)k, k, rank)], 1u);
}

template <typename T>
cudaError_t dalloc(T **p, size_t count) {
  return cudaMalloc((void **)p, std::max<size_t>(count, 1) * sizeof(T));
}

// Bytes of shared memory a thread-per-edge CTA needs at out-degree bound d.
size_t sample_smem(uint32_t d) { return (size_t)d * 12; }

}  // namespace

struct kclpp_sampling {
  const kclpp_graph *g = nullptr;
  int device = 0;
  int k = 0;
  uint32_t n = 0;
  uint64_t target = 0, seed = 0, total = 0, sampled = 0, threshold = 0, cap = 0;
  double prob = 1.0;
  int all = 1;
  uint32_t waves = 1, passes = 0;
  uint32_t *d_rows = nullptr;
  uint8_t *d_wave = nullptr;
  uint32_t *d_rho = nullptr, *d_rank = nullptr, *d_push = nullptr, *d_order = nullptr;
  uint2 *d_vals = nullptr;              // three buffers of n pairs
  unsigned long long *d_keys = nullptr; // n
  PrefixBest *d_best = nullptr;
  OrderScratch ord;
  std::vector<unsigned long long> wave_at;  // first row of each wave, then the sample's end
  ~kclpp_sampling() {
    cudaSetDevice(device);
    for (void *p : {(void *)d_rows, (void *)d_wave, (void *)d_rho, (void *)d_vals, (void *)d_rank, (void *)d_push,
                    (void *)d_order, (void *)d_keys, (void *)d_best})
      if (p) cudaFree(p);
    order_scratch_free(ord);
  }
};

namespace {

template <int K>
kclpp_status launch_groups(kclpp_ctx *c, kclpp_sampling *S, const SampleArgs &base, const uint32_t *d_roots,
                           const uint32_t (&bounds)[5], const uint32_t (&dmax)[4], uint32_t *d_work) {
  cudaStream_t st = ctx_stream(c);
  const int sms = ctx_sms(c);
  int optin = 0;
  SCUDA(cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, S->device));
  const size_t limit = (size_t)optin - 256;  // room for the static counters
  auto wide = k_sample<K>;
  auto warps = k_sample_warps<K>;
  SCUDA(cudaFuncSetAttribute(wide, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)limit));
  SCUDA(cudaFuncSetAttribute(warps, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)limit));
  // The slab is freed on every return path (cudaFree waits for the kernels).
  struct Slab {
    uint32_t *p = nullptr;
    ~Slab() {
      if (p) cudaFree(p);
    }
  } slab;
  for (int grp = 0; grp < 4; ++grp) {
    const uint32_t lo = bounds[grp], hi = bounds[grp + 1];
    if (lo == hi) continue;
    SampleArgs a = base;
    a.roots = d_roots + lo;
    a.num_roots = hi - lo;
    a.dmax = dmax[grp];
    a.ws = (a.dmax + 31) / 32;
    a.work = d_work + grp;
    const bool slabbed = grp == 0;
    const int threads = slabbed ? kSampleThreads : kGroupThreads[grp - 1];
    const size_t smem = slabbed ? sample_smem(a.dmax) : warp_layout(a.dmax, threads / 32).total;
    int per_sm = 0;
    SCUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, slabbed ? wide : warps, threads, smem));
    if (per_sm < 1) return set_error(KCLPP_ERR_UNSUPPORTED, "sampling kernel does not fit (%zu B shared)", smem);
    const uint32_t grid = std::min<uint32_t>((uint32_t)per_sm * (uint32_t)sms, a.num_roots);
    if (slabbed) {
      a.slab_words = (uint64_t)a.dmax * a.ws;
      SCUDA(dalloc(&slab.p, (size_t)grid * a.slab_words));
      a.slab = slab.p;
      wide<<<grid, threads, smem, st>>>(a);
    } else {
      warps<<<grid, threads, smem, st>>>(a);
    }
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return set_error(KCLPP_ERR_CUDA, "sampling kernel: %s", cudaGetErrorString(e));
    ctx_count_launch(c, 1);
  }
  cudaError_t e = cudaStreamSynchronize(st);
  if (e != cudaSuccess) return set_error(KCLPP_ERR_CUDA, "sampling kernel: %s", cudaGetErrorString(e));
  return KCLPP_OK;
}

kclpp_status launch_k(int k, kclpp_ctx *c, kclpp_sampling *S, const SampleArgs &a, const uint32_t *d_roots,
                      const uint32_t (&bounds)[5], const uint32_t (&dmax)[4], uint32_t *d_work) {
  switch (k) {
    case 3: return launch_groups<3>(c, S, a, d_roots, bounds, dmax, d_work);
    case 4: return launch_groups<4>(c, S, a, d_roots, bounds, dmax, d_work);
    case 5: return launch_groups<5>(c, S, a, d_roots, bounds, dmax, d_work);
    case 6: return launch_groups<6>(c, S, a, d_roots, bounds, dmax, d_work);
    case 7: return launch_groups<7>(c, S, a, d_roots, bounds, dmax, d_work);
    case 8: return launch_groups<8>(c, S, a, d_roots, bounds, dmax, d_work);
    default: return set_error(KCLPP_ERR_UNSUPPORTED, "k = %d", k);
  }
}

// The kept rows grouped by wave, in buffers of their number.  Where the device
// has no room for a second copy of them, they are drawn again in place:
// redraw(at) samples with every row at the cursor of its wave.
template <typename Redraw>
kclpp_status group_by_wave(kclpp_ctx *c, kclpp_sampling *S, Redraw &&redraw) {
  S->wave_at.assign(smp::kMaxWaves + 1, 0);
  if (!S->sampled) return KCLPP_OK;
  cudaStream_t st = ctx_stream(c);
  struct Tmp {
    unsigned long long *cnt = nullptr;
    uint32_t *rows = nullptr;
    uint8_t *wave = nullptr;
    ~Tmp() { cudaFree(cnt); cudaFree(rows); cudaFree(wave); }
  } t;
  const size_t words = smp::kMaxWaves + 1;
  SCUDA(dalloc(&t.cnt, words));
  cudaError_t room = dalloc(&t.rows, (size_t)S->sampled * S->k);
  if (room == cudaSuccess) room = dalloc(&t.wave, (size_t)S->sampled);
  if (room == cudaErrorMemoryAllocation) cudaGetLastError();
  else SCUDA(room);
  SCUDA(cudaMemsetAsync(t.cnt, 0, words * 8, st));
  const uint32_t grid = (uint32_t)std::min<uint64_t>((S->sampled + 2047) / 2048, (uint64_t)ctx_sms(c) * 8);
  k_wave_count<<<grid, 256, 0, st>>>(S->d_wave, S->sampled, t.cnt);
  SCUDA(cudaGetLastError());
  SCUDA(cudaMemcpyAsync(S->wave_at.data(), t.cnt, words * 8, cudaMemcpyDeviceToHost, st));
  SCUDA(cudaStreamSynchronize(st));
  for (size_t w = 1; w < words; ++w) S->wave_at[w] += S->wave_at[w - 1];
  SCUDA(cudaMemcpyAsync(t.cnt, S->wave_at.data(), words * 8, cudaMemcpyHostToDevice, st));
  if (room != cudaSuccess) {
    ctx_count_launch(c, 1);
    cudaFree(t.rows);  // the redraw may need a slab
    t.rows = nullptr;
    return redraw(t.cnt);
  }
  k_wave_move<<<grid, 256, 0, st>>>(S->d_rows, S->d_wave, S->sampled, S->k, t.cnt, t.rows, t.wave);
  SCUDA(cudaGetLastError());
  SCUDA(cudaStreamSynchronize(st));
  ctx_count_launch(c, 2);
  std::swap(S->d_rows, t.rows);
  std::swap(S->d_wave, t.wave);
  return KCLPP_OK;
}

// Runs the sampling kernel until the row buffer holds every kept clique (a
// second run, with the buffer sized to the first run's count, only when the
// first overflowed; the kept set does not change between runs).
kclpp_status sample(kclpp_ctx *c, kclpp_sampling *S) {
  const HostDag &D = graph_dag(S->g);
  const int k = S->k;
  // The graph's counting schedule lists every root by decreasing out-degree;
  // the launch groups are ranges of it, ending where k - 1 no longer fits.
  uint32_t bounds[5] = {0, 0, 0, 0, 0}, dmax[4] = {0, 0, 0, 0};
  for (uint32_t v = 0; v < D.n; ++v) {
    const uint32_t d = (uint32_t)(D.off[v + 1] - D.off[v]);
    if (d < (uint32_t)(k - 1)) continue;
    const int grp = d > kWarpRoots ? 0 : d > kGroupDeg[0] ? 1 : d > kGroupDeg[1] ? 2 : 3;
    ++bounds[grp + 1];
    dmax[grp] = std::max(dmax[grp], d);
  }
  for (int i = 1; i < 5; ++i) bounds[i] += bounds[i - 1];
  if (!bounds[4] || S->total == 0) {
    S->sampled = 0;
    S->wave_at.assign(smp::kMaxWaves + 1, 0);
    return KCLPP_OK;
  }
  cudaStream_t st = ctx_stream(c);
  uint32_t *d_work = nullptr;
  unsigned long long *d_count = nullptr;
  auto release = [&]() {
    if (d_work) cudaFree(d_work);
    if (d_count) cudaFree(d_count);
  };
  // One run of the kernels into S's buffers; *got receives the rows counted.
  auto draw = [&](unsigned long long *wave_at, unsigned long long *got) -> kclpp_status {
    SCUDA(cudaMemsetAsync(d_work, 0, 16, st));
    SCUDA(cudaMemsetAsync(d_count, 0, 8, st));
    SampleArgs a{};
    a.off = graph_dev_offsets(S->g);
    a.cols = graph_dev_cols(S->g);
    a.seed = S->seed;
    a.threshold = S->threshold;
    a.all = S->all;
    a.waves = S->waves;
    a.rows = S->d_rows;
    a.wave = S->d_wave;
    a.cap = S->cap;
    a.count = d_count;
    a.wave_at = wave_at;
    a.bit_rows = graph_dev_bit_rows(S->g);
    a.bits = graph_dev_bits(S->g);
    STRY(launch_k(k, c, S, a, graph_dev_count_roots(S->g), bounds, dmax, d_work));
    SCUDA(cudaMemcpyAsync(got, d_count, 8, cudaMemcpyDeviceToHost, st));
    SCUDA(cudaStreamSynchronize(st));
    return KCLPP_OK;
  };
  kclpp_status status = KCLPP_OK;
  for (int attempt = 0; attempt < 2; ++attempt) {
    cudaError_t e = cudaSuccess;
    if (e == cudaSuccess && !d_work) e = dalloc(&d_work, 4);
    if (e == cudaSuccess && !d_count) e = dalloc(&d_count, 1);
    if (e == cudaSuccess && !S->d_rows) e = dalloc(&S->d_rows, (size_t)S->cap * k);
    if (e == cudaSuccess && !S->d_wave) e = dalloc(&S->d_wave, (size_t)S->cap);
    if (e != cudaSuccess) {
      release();
      return set_error(e == cudaErrorMemoryAllocation ? KCLPP_ERR_NOMEM : KCLPP_ERR_CUDA, "sampling: %s",
                       cudaGetErrorString(e));
    }
    unsigned long long got = 0;
    status = draw(nullptr, &got);
    if (status != KCLPP_OK) break;
    S->sampled = got;
    if (got <= S->cap) break;
    if (attempt == 1) {
      status = set_error(KCLPP_ERR_CUDA, "sampling: the kept set changed between runs");
      break;
    }
    cudaFree(S->d_rows);
    cudaFree(S->d_wave);
    S->d_rows = nullptr;
    S->d_wave = nullptr;
    S->cap = got;
  }
  if (status == KCLPP_OK)
    status = group_by_wave(c, S, [&](unsigned long long *wave_at) {
      unsigned long long none = 0;
      return draw(wave_at, &none);
    });
  release();
  return status;
}

kclpp_status check_ctx(kclpp_ctx *c, const kclpp_sampling *S) {
  if (!c || !S) return set_error(KCLPP_ERR_INVALID, "null argument");
  if (ctx_device(c) != S->device) return set_error(KCLPP_ERR_INVALID, "context and sampling on different devices");
  SCUDA(cudaSetDevice(S->device));
  return KCLPP_OK;
}

template <int K>
void launch_wave(const kclpp_sampling *S, uint32_t w, int sms, const uint2 *in, uint2 *out, uint2 *clear,
                 cudaStream_t st) {
  const uint64_t lo = S->wave_at[w], hi = S->wave_at[w + 1], work = std::max<uint64_t>(hi - lo, S->n);
  const uint32_t grid = (uint32_t)std::min<uint64_t>((work + kPassThreads - 1) / kPassThreads, (uint64_t)sms * 8);
  k_wave<K><<<grid, kPassThreads, 0, st>>>(S->d_rows, lo, hi, S->n, in, out, clear);
}

kclpp_status run_passes(kclpp_ctx *c, kclpp_sampling *S, uint32_t passes) {
  if (!passes || !S->sampled || !S->n) return KCLPP_OK;
  cudaStream_t st = ctx_stream(c);
  const int sms = ctx_sms(c);
  const size_t n = S->n;
  if (!S->d_vals) SCUDA(dalloc(&S->d_vals, 3 * n));
  uint2 *b[3] = {S->d_vals, S->d_vals + n, S->d_vals + 2 * n};
  const uint32_t grid_n = (S->n + kPassThreads - 1) / kPassThreads;
  k_open<<<grid_n, kPassThreads, 0, st>>>(S->n, S->d_rho, b[0], b[1], b[2]);
  uint64_t step = 0;
  for (uint32_t p = 0; p < passes; ++p) {
    for (uint32_t w = 0; w < S->waves; ++w, ++step) {
      const uint2 *in = b[step % 3];
      uint2 *out = b[(step + 1) % 3], *clear = b[(step + 2) % 3];
      switch (S->k) {
        case 3: launch_wave<3>(S, w, sms, in, out, clear, st); break;
        case 4: launch_wave<4>(S, w, sms, in, out, clear, st); break;
        case 5: launch_wave<5>(S, w, sms, in, out, clear, st); break;
        case 6: launch_wave<6>(S, w, sms, in, out, clear, st); break;
        case 7: launch_wave<7>(S, w, sms, in, out, clear, st); break;
        default: launch_wave<8>(S, w, sms, in, out, clear, st); break;
      }
    }
    SCUDA(cudaGetLastError());
    ctx_count_launch(c, (int)S->waves);
  }
  k_close<<<grid_n, kPassThreads, 0, st>>>(S->n, b[step % 3], S->d_rho);
  SCUDA(cudaGetLastError());
  ctx_count_launch(c, 2);
  SCUDA(cudaStreamSynchronize(st));
  return KCLPP_OK;
}

}  // namespace

extern "C" {

kclpp_status kclpp_sampling_create(kclpp_ctx *c, const kclpp_graph *g, int k, uint64_t target, uint64_t seed,
                                   uint32_t waves, kclpp_sampling **out) {
  if (!c || !g || !out) return set_error(KCLPP_ERR_INVALID, "null argument");
  *out = nullptr;
  if (k < 3 || k > KCLPP_MAX_K)
    return set_error(KCLPP_ERR_UNSUPPORTED, "k = %d outside the sampling range [3, %d]", k, KCLPP_MAX_K);
  if (target < 1 || target > 0x7fffffffull) return set_error(KCLPP_ERR_INVALID, "target outside [1, 2^31 - 1]");
  if (waves < 1 || waves > smp::kMaxWaves) return set_error(KCLPP_ERR_INVALID, "waves outside [1, 256]");
  if (ctx_device(c) != graph_device(g)) return set_error(KCLPP_ERR_INVALID, "context and graph on different devices");
  const HostDag &D = graph_dag(g);
  if (D.core > smp::kMaxDegree)
    return set_error(KCLPP_ERR_UNSUPPORTED, "out-degree %u exceeds %u", D.core, smp::kMaxDegree);
  std::unique_ptr<kclpp_sampling> S(new kclpp_sampling());
  S->g = g;
  S->device = ctx_device(c);
  S->k = k;
  S->n = D.n;
  S->target = target;
  S->seed = seed;
  S->waves = waves;
  SCUDA(cudaSetDevice(S->device));
  // The COUNT task (kCDensestSamplingKclistpp.c:153-157, 191-195), then p (:272).
  STRY(kclpp_count_cliques(c, g, k, nullptr, &S->total));
  S->all = target >= S->total;
  S->prob = S->all ? 1.0 : (double)target / (double)S->total;
  S->threshold = S->all ? 0 : (uint64_t)std::ldexp(S->prob, 64);
  // Room for the expected sample plus a margin well beyond its spread.
  S->cap = S->all ? S->total : std::min<uint64_t>(S->total, target + target / 8 + 4096);
  SCUDA(dalloc(&S->d_rho, S->n));
  SCUDA(dalloc(&S->d_rank, S->n));
  SCUDA(dalloc(&S->d_push, S->n));
  cudaStream_t st = ctx_stream(c);
  SCUDA(cudaMemsetAsync(S->d_rho, 0, (size_t)std::max<uint32_t>(S->n, 1) * 4, st));
  STRY(sample(c, S.get()));
  *out = S.release();
  return KCLPP_OK;
}

void kclpp_sampling_free(kclpp_sampling *s) { delete s; }

kclpp_status kclpp_sampling_info_get(const kclpp_sampling *s, kclpp_sampling_info *info) {
  if (!s || !info) return set_error(KCLPP_ERR_INVALID, "null argument");
  info->cliques_total = s->total;
  info->sampled = s->sampled;
  info->prob = s->prob;
  info->threshold = s->threshold;
  info->all = s->all;
  info->waves = s->waves;
  info->passes = s->passes;
  return KCLPP_OK;
}

kclpp_status kclpp_sampling_cliques(kclpp_ctx *c, const kclpp_sampling *s, uint32_t *rows, uint8_t *waves) {
  STRY(check_ctx(c, s));
  const int k = s->k;
  const size_t S = (size_t)s->sampled;
  if (!S || (!rows && !waves)) return KCLPP_OK;
  std::vector<uint32_t> r(S * k);
  std::vector<uint8_t> w(S);
  cudaStream_t st = ctx_stream(c);
  SCUDA(cudaMemcpyAsync(r.data(), s->d_rows, r.size() * 4, cudaMemcpyDeviceToHost, st));
  SCUDA(cudaMemcpyAsync(w.data(), s->d_wave, S, cudaMemcpyDeviceToHost, st));
  SCUDA(cudaStreamSynchronize(st));
  std::vector<size_t> idx(S);
  std::iota(idx.begin(), idx.end(), (size_t)0);
  std::sort(idx.begin(), idx.end(), [&](size_t a, size_t b) {
    for (int j = k - 1; j >= 0; --j)
      if (r[a * k + j] != r[b * k + j]) return r[a * k + j] < r[b * k + j];
    return false;
  });
  for (size_t i = 0; i < S; ++i) {
    if (rows) memcpy(rows + i * k, &r[idx[i] * k], (size_t)k * 4);
    if (waves) waves[i] = w[idx[i]];
  }
  return KCLPP_OK;
}

kclpp_status kclpp_sampling_passes(kclpp_ctx *c, kclpp_sampling *s, uint32_t passes) {
  STRY(check_ctx(c, s));
  STRY(run_passes(c, s, passes));
  s->passes += passes;
  return KCLPP_OK;
}

kclpp_status kclpp_sampling_get_rho(kclpp_ctx *c, const kclpp_sampling *s, uint32_t *rho) {
  STRY(check_ctx(c, s));
  if (!s->n) return KCLPP_OK;
  if (!rho) return set_error(KCLPP_ERR_INVALID, "null argument");
  cudaStream_t st = ctx_stream(c);
  SCUDA(cudaMemcpyAsync(rho, s->d_rho, (size_t)s->n * 4, cudaMemcpyDeviceToHost, st));
  SCUDA(cudaStreamSynchronize(st));
  return KCLPP_OK;
}

kclpp_status kclpp_sampling_set_rho(kclpp_ctx *c, kclpp_sampling *s, const uint32_t *rho, uint32_t passes) {
  STRY(check_ctx(c, s));
  if (s->n && !rho) return set_error(KCLPP_ERR_INVALID, "null argument");
  cudaStream_t st = ctx_stream(c);
  if (s->n) SCUDA(cudaMemcpyAsync(s->d_rho, rho, (size_t)s->n * 4, cudaMemcpyHostToDevice, st));
  SCUDA(cudaStreamSynchronize(st));
  s->passes = passes;
  return KCLPP_OK;
}

kclpp_status kclpp_sampling_extract(kclpp_ctx *c, kclpp_sampling *s, uint32_t T, kclpp_sampling_report *rep,
                                    uint32_t *order) {
  STRY(check_ctx(c, s));
  if (!rep) return set_error(KCLPP_ERR_INVALID, "null argument");
  if (T < 1) return set_error(KCLPP_ERR_INVALID, "T must be at least 1");
  memset(rep, 0, sizeof *rep);
  rep->T = T;
  const uint32_t n = s->n;
  const int k = s->k;
  if (!n) return KCLPP_OK;
  cudaStream_t st = ctx_stream(c);
  std::vector<uint32_t> rho(n), ord(n), rank(n);
  SCUDA(cudaMemcpyAsync(rho.data(), s->d_rho, (size_t)n * 4, cudaMemcpyDeviceToHost, st));
  SCUDA(cudaStreamSynchronize(st));
  uint32_t top = 0;
  for (uint32_t i = 0; i < n; ++i) top |= rho[i];
  // Vertices by decreasing load, ties by ascending id (:367-373); each kept
  // clique to its last vertex in that order (:375-383); the densest prefix, the
  // first strictly best count / size (:385-394).
  SCUDA(order_scratch_make(s->ord, n));
  if (!s->d_order) SCUDA(dalloc(&s->d_order, n));
  if (!s->d_keys) SCUDA(dalloc(&s->d_keys, n));
  if (!s->d_best) SCUDA(dalloc(&s->d_best, 1));
  uint64_t launched = 0;
  SCUDA(order_by_key32(s->d_rho, n, top, s->ord, s->d_keys, s->d_order, s->d_rank, st, &launched));
  SCUDA(cudaMemsetAsync(s->d_push, 0, (size_t)n * 4, st));
  if (s->sampled) {
    const uint32_t grid =
        (uint32_t)std::min<uint64_t>((s->sampled + kPassThreads - 1) / kPassThreads, (uint64_t)ctx_sms(c) * 8);
    k_push<<<grid, kPassThreads, 0, st>>>(s->d_rows, s->sampled, k, s->d_rank, s->d_push);
    SCUDA(cudaGetLastError());
    ++launched;
  }
  SCUDA(densest_prefix32(s->d_push, n, s->ord, s->d_best, st, &launched));
  ctx_count_launch(c, (int)launched);
  PrefixBest best;
  SCUDA(cudaMemcpyAsync(&best, s->d_best, sizeof best, cudaMemcpyDeviceToHost, st));
  SCUDA(cudaMemcpyAsync(ord.data(), s->d_order, (size_t)n * 4, cudaMemcpyDeviceToHost, st));
  SCUDA(cudaMemcpyAsync(rank.data(), s->d_rank, (size_t)n * 4, cudaMemcpyDeviceToHost, st));
  SCUDA(cudaStreamSynchronize(st));
  rep->n = best.n;
  rep->m = best.cliques;
  rep->density = best.density;
  // The bound from the loads (:400-417), in the reference's operation order.
  {
    uint64_t sum = 0;
    double ub = 0, ip1ck = 0;
    for (uint32_t i = 0; i < n; ++i) {
      sum += rho[ord[i]];
      if (i + 1 == (uint32_t)k) ip1ck = 1;
      else if (i + 1 > (uint32_t)k) ip1ck = (ip1ck * (double)(i + 1)) / (double)(i + 1 - k);
      const double avg = (double)sum / (double)T;
      if (ip1ck < avg) {
        ub = ip1ck / (double)(i + 1);
      } else {
        const double v = avg / (double)(i + 1);
        if (ub < v) ub = v;
        break;
      }
    }
    rep->ub = ub;
  }
  // The densest subgraph's exact clique count (MakeDensestSubgraphEdgeList and
  // the COUNT_IN_SUBGRAPH task, :420-435, :467-471): its edges, labelled by
  // their position in the order, through the library's own pipeline.
  const HostDag &D = graph_dag(s->g);
  std::vector<uint32_t> pairs;
  std::vector<uint32_t> inside(ord.begin(), ord.begin() + rep->n);
  std::sort(inside.begin(), inside.end());
  for (uint32_t a : inside) {
    for (uint64_t e = D.off[a]; e < D.off[a + 1]; ++e) {
      const uint32_t b = D.cols[e];
      if (rank[b] >= rep->n) continue;
      pairs.push_back(rank[a]);
      pairs.push_back(rank[b]);
    }
  }
  rep->sub_e = pairs.size() / 2;
  if (rep->sub_e) {
    kclpp_edge_list *el = nullptr;
    kclpp_graph *sg = nullptr;
    kclpp_status st2 = kclpp_edge_list_create(pairs.data(), rep->sub_e, &el);
    // size, core value and count are those of any degeneracy order
    if (st2 == KCLPP_OK) st2 = kclpp_build_graph_mode(c, el, KCLPP_ORDER_FAST, &sg);
    if (st2 == KCLPP_OK) st2 = kclpp_count_cliques(c, sg, k, nullptr, &rep->sub_cliques);
    uint32_t sn = 0, score = 0;
    uint64_t sm = 0;
    if (st2 == KCLPP_OK) st2 = kclpp_graph_info(sg, &sn, &sm, &score);
    kclpp_graph_free(sg);
    kclpp_edge_list_free(el);
    if (st2 != KCLPP_OK) return st2;
    rep->sub_n = sn;
    rep->sub_core = score;
  }
  // The report line's figures (:475-477), with the reference's unsigned n - 1.
  rep->edge_density = (double)rep->sub_e * 2.0 / (double)rep->sub_n / (double)(uint32_t)(rep->sub_n - 1u);
  rep->clique_density = (double)rep->sub_cliques / (double)rep->sub_n;
  rep->upper_bound = rep->ub / s->prob / (1 - std::sqrt(6 * std::log((double)n) / rep->ub));
  if (order) memcpy(order, ord.data(), (size_t)n * 4);
  return KCLPP_OK;
}

kclpp_status kclpp_sampling_main(kclpp_ctx *c, const kclpp_graph *g, int k, uint32_t num_iter, uint64_t target,
                                 uint64_t seed, uint32_t waves, kclpp_sampling_report *reps, int cap, int *count) {
  if (count) *count = 0;
  if (cap > 0 && !reps) return set_error(KCLPP_ERR_INVALID, "null argument");
  kclpp_sampling *s = nullptr;
  STRY(kclpp_sampling_create(c, g, k, target, seed, waves, &s));
  std::unique_ptr<kclpp_sampling> hold(s);
  int made = 0;
  for (uint64_t T = 1; T <= num_iter; T <<= 1) {
    STRY(kclpp_sampling_passes(c, s, (uint32_t)T - s->passes));
    if (made < cap) STRY(kclpp_sampling_extract(c, s, (uint32_t)T, &reps[made], nullptr));
    ++made;
  }
  if (count) *count = std::min(made, std::max(cap, 0));
  return KCLPP_OK;
}

}  // extern "C"
