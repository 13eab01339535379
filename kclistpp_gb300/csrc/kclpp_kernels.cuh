// kclpp_kernels.cuh -- the clique kernels (included by one translation unit per mode).
//
// Three modes share one root-vertex skeleton (build G_s as bitmaps, then work
// per row / per root edge):
//
//  MODE_COUNT  k-clique degree of every vertex (onepass/recursion,
//              kClistCoreTrim.c:368-416).  Rows are the symmetric adjacency S
//              of G_s; the (k-1)-cliques of G_s through x number the
//              (k-2)-cliques of S[x], counted with the id orientation
//              A[y] = S[y] ∩ {ids below y}, popcount at the last level.
//
//  MODE_ORDER  cliques credited to their smallest-key member (Sim-kClist++'s
//              rho_add, kCDensestCmpSync.c:138-146; PAVA's largest level,
//              kCDensestNoAtom.c:191-213).  G_s is relabelled by key rank and
//              oriented upward: the cliques whose smallest member in G_s is p
//              number the (k-2)-cliques of Up[p]; p takes them if its key is
//              below s's, otherwise s does.  Pure popcount counting: no clique
//              is visited one by one.
//
//  MODE_SEQ    Seq-kClist++'s in-place "++" chain (kCDensestNoAtom.c:155-268),
//              one independent stream per root edge (s, t) starting from the
//              pass-start r.  Cliques are visited in the reference's order
//              (ascending ids at every level); the argmin prefix is cached as a
//              vertex and its value re-read at every comparison, exactly as the
//              reference does.  At the last level the chain
//                  for v in V ascending: if cur[v] < cur[g] then cur[v]++ else cur[g]++
//              runs 32 candidates at a time (tiers M, L): a candidate fails
//              (credits g) iff cur[v] >= c0 + (failures before it); the failure
//              mask is the unique fixed point of that rule and is found by
//              iterating ballots (lane i is final after i+1 rounds, so the loop
//              is bounded by 33 rounds).  With rows in shared memory the last
//              two levels are first settled 32 vertices at a time by counting
//              (TinyStream: at most 64 candidates, in registers; PairLevel:
//              the others), and only a group whose comparisons can still
//              change runs its chains one after another.
//
// Set iteration always walks a copy of the set (`it`) and intersects with the
// unmodified set, because the child set of u is P ∩ N+(u) over all of P.
#pragma once

#include <algorithm>
#include <mutex>
#include <type_traits>
#include <utility>
#include <vector>

#include "kclpp_dev.cuh"

namespace kclpp {
namespace dev {

// ========================================================================
// Tier S: one warp per root, d <= 64, 64-bit rows, one lane per row / edge.
constexpr int kSMaxD = 64;
constexpr int kSDl = kSMaxD + 1;  // per-lane delta stride
constexpr int kSFew = 32;         // most members of a root whose rows are built in registers

// A root's members by id: an open-addressing table of 2^bits slots, at most a
// quarter full up to 512 members and half full beyond.  An id's home is the
// top bits of its multiplicative hash (a trimmed core's members are runs of
// consecutive ids, which an identity hash would chain together); a slot holds
// 20 other hash bits and the member's list position.  The induced rows look
// every out-neighbour of every member up: a probe or two replaces a binary
// search of the list (~9 dependent shared-memory reads at 500 members).
__host__ __device__ __forceinline__ int tab_bits(uint32_t d) {
  int b = 6;
  while ((1u << b) < 4 * d && ((1u << b) < 2048 || (1u << b) < 2 * d)) ++b;
  return b;
}
constexpr uint32_t kTabEmpty = 0xffffffffu;  // no entry: positions stay below 4095
__device__ __forceinline__ void tab_insert(uint32_t *tab, int bits, uint32_t y, int pos) {
  const uint32_t h = y * 0x9E3779B1u, mask = (1u << bits) - 1u, e = (h << 12) | (uint32_t)pos;
  uint32_t at = h >> (32 - bits);
  while (atomicCAS(tab + at, kTabEmpty, e) != kTabEmpty) at = (at + 1) & mask;
}
// Position of y in list, or -1.
__device__ __forceinline__ int tab_find(const uint32_t *tab, int bits, const uint32_t *list, uint32_t y) {
  const uint32_t h = y * 0x9E3779B1u, mask = (1u << bits) - 1u;
  for (uint32_t at = h >> (32 - bits);; at = (at + 1) & mask) {
    const uint32_t e = tab[at];
    if (e == kTabEmpty) return -1;
    if (((e >> 12) ^ h) << 12 == 0 && list[e & 4095u] == y) return (int)(e & 4095u);
  }
}

// A vertex's bitmap row, if it has one: the word its out-neighbours' bits start
// at in a.bits, the id of the first bit and the number of ids it covers.
constexpr uint32_t kNoBitRow = 0xffffffffu;
__device__ __forceinline__ uint4 bit_row(const PassArgs &a, uint32_t x) {
  return a.bit_rows ? __ldg(a.bit_rows + x) : make_uint4(kNoBitRow, 0u, 0u, 0u);
}
// Bit of id y in the row starting at word `row`, id `first`, `span` ids long.
__device__ __forceinline__ bool bit_at(const PassArgs &a, uint32_t row, uint32_t first, uint32_t span, uint32_t y) {
  const uint32_t t = y - first;
  return t < span && ((__ldg(a.bits + row + (t >> 5)) >> (t & 31)) & 1u);
}

// Shared-memory add of a 64-bit word by its native 32-bit halves (the 64-bit
// form is a compare-and-swap loop, which serialises when warps meet in a word).
__device__ __forceinline__ void shared_add(unsigned long long *p, unsigned long long x) {
  uint32_t *w = reinterpret_cast<uint32_t *>(p);
  const uint32_t lo = (uint32_t)x;
  const uint32_t hi = (uint32_t)(x >> 32) + (atomicAdd(w, lo) + lo < lo);
  if (hi) atomicAdd(w + 1, hi);
}
template <int MODE>
struct SmemS {
  uint32_t list[kSMaxD];
  uint32_t tab[4 * kSMaxD];
  unsigned long long rows[kSMaxD];
  unsigned long long base[kSMaxD + 1];  // SEQ: pass-start r; ORDER: keys
  unsigned long long acc[kSMaxD + 1];   // SEQ: per-root increments
  uint8_t rank[kSMaxD];
  uint8_t inv[kSMaxD];
  uint32_t dl[MODE == MODE_SEQ ? 32 * kSDl : 1];  // SEQ: per-lane stream deltas
};

__device__ __forceinline__ unsigned long long below64(int y) {
  return y == 0 ? 0ull : ((1ull << y) - 1ull);
}

// Number of R-cliques inside P.  Orientation rows[y], restricted to ids below
// y when BELOW (symmetric rows), used as is otherwise (upward rows).
template <int R, bool BELOW>
__device__ __forceinline__ uint64_t cnt64(unsigned long long P, const unsigned long long *rows) {
  if constexpr (R == 0) {
    return 1;
  } else if constexpr (R == 1) {
    return (uint64_t)__popcll(P);
  } else {
    uint64_t c = 0;
    unsigned long long it = P;
    while (it) {
      const int y = __ffsll((long long)it) - 1;
      it &= it - 1;
      unsigned long long A = rows[y];
      if (BELOW) A &= below64(y);
      c += cnt64<R - 1, BELOW>(P & A, rows);
    }
    return c;
  }
}

// Seq chain inside one lane (tier S).  L = levels left (k-2 at the top).
// Returns the number of cliques visited.
template <int L>
__device__ __forceinline__ uint32_t seq64(unsigned long long P, int g, const unsigned long long *rows,
                                          const unsigned long long *base, uint32_t *dl) {
  if constexpr (L == 1) {
    // clique_size == 3 branch, kCDensestNoAtom.c:162-171
    uint32_t c = 0;
    unsigned long long it = P;
    while (it) {
      const int u = __ffsll((long long)it) - 1;
      it &= it - 1;
      const int g2 = (base[u] + dl[u]) < (base[g] + dl[g]) ? u : g;
      dl[g2]++;
      ++c;
    }
    return c;
  } else if constexpr (L == 2) {
    // l == 2 branch, kCDensestNoAtom.c:173-188
    uint32_t c = 0;
    unsigned long long it = P;
    while (it) {
      const int u = __ffsll((long long)it) - 1;
      it &= it - 1;
      const int g2 = (base[u] + dl[u]) < (base[g] + dl[g]) ? u : g;
      unsigned long long V = P & rows[u];
      while (V) {
        const int v = __ffsll((long long)V) - 1;
        V &= V - 1;
        const int g3 = (base[v] + dl[v]) < (base[g2] + dl[g2]) ? v : g2;
        dl[g3]++;
        ++c;
      }
    }
    return c;
  } else {
    // general level, kCDensestNoAtom.c:218-267
    if (__popcll(P) < L) return 0;
    uint32_t c = 0;
    unsigned long long it = P;
    while (it) {
      const int u = __ffsll((long long)it) - 1;
      it &= it - 1;
      const int g2 = (base[u] + dl[u]) < (base[g] + dl[g]) ? u : g;
      c += seq64<L - 1>(P & rows[u], g2, rows, base, dl);
    }
    return c;
  }
}

// IDENT = true: the schedule is every vertex in id order (no root list), a
// vertex being a root of this launch when its out-degree lies in
// [a.deg_lo, a.deg_hi]; the roots' own clique counts are also summed into
// *a.total.  Used by the entry point that allocates nothing.
template <int MODE, int K, bool IDENT = false>
__global__ void __launch_bounds__(kWarpsS * 32) tier_s_kernel(PassArgs a) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  using SM = SmemS<MODE>;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  SM &sm = reinterpret_cast<SM *>(smem_raw)[wid];
  if constexpr (MODE == MODE_SEQ) {
    for (int i = lane; i <= kSMaxD; i += 32) sm.acc[i] = 0;
    for (int i = 0; i < kSDl; ++i) sm.dl[lane * kSDl + i] = 0;
  }
  __syncwarp();
  for (;;) {
    uint32_t idx = 0;
    if (lane == 0) idx = atomicAdd(a.work, 1u);
    idx = __shfl_sync(KCL_FULL, idx, 0);
    if (idx >= a.num_roots) break;
    const uint32_t s = IDENT ? idx : a.roots[idx];
    uint64_t o;
    int d;
    const uint32_t *lcols;
    root_span(a, s, o, d, lcols);
    if constexpr (IDENT) {
      if ((uint32_t)d < a.deg_lo || (uint32_t)d > a.deg_hi) continue;
    }
    if (d > kSMaxD) {
      if (lane == 0) atomicOr(a.err, ERR_DEGREE);
      continue;
    }
    if (d < K - 1 || d == 0) continue;
    for (int i = lane; i < d; i += 32) sm.list[i] = lcols[o + i];
    int tau = 0;
    if constexpr (MODE == MODE_ORDER) {
      for (int i = lane; i < d; i += 32) sm.base[i] = vertex_key(a, sm.list[i]);
      const uint64_t ks = vertex_key(a, s);
      __syncwarp();
      int t = 0;
      for (int i = lane; i < d; i += 32) {
        const uint64_t ki = sm.base[i];
        int r = 0;
        for (int j = 0; j < d; ++j) {
          const uint64_t kj = sm.base[j];
          r += (kj < ki) || (kj == ki && j < i);
        }
        sm.rank[i] = (uint8_t)r;
        sm.inv[r] = (uint8_t)i;
        t += (ki <= ks);  // (key_i, i) < (key_s, d): s has the largest id
      }
      tau = warp_sum(t);
    }
    if constexpr (MODE == MODE_SEQ) {
      // Shared loads: the root's values as the load vector holds them now.
      if (a.shared_loads) {
        for (int i = lane; i < d; i += 32) sm.base[i] = __ldcg(a.out + sm.list[i]);
        if (lane == 0) sm.base[d] = __ldcg(a.out + s);
      } else {
        for (int i = lane; i < d; i += 32) sm.base[i] = a.r_in[sm.list[i]];
        if (lane == 0) sm.base[d] = a.r_in[s];
      }
    }
    for (int i = lane; i < kSMaxD; i += 32) sm.rows[i] = 0;
    __syncwarp();
    if (K >= 3 && d <= kSFew) {
      // Rows as below, of at most a word: row `lane` in a register.  A member
      // with a bitmap row is asked about the ones before it; another's out-list
      // is merged with the members, four neighbours at a time.  Instruction
      // issue over many small roots bounds this, and the table, its look-ups and
      // a step per member without a row cost more than these roots hold: 400,000
      // vertices of out-degree <= 37, a k = 3 Sim pass 427 us with the table, 322
      // so; an RMAT-18 graph, whose hubs the bitmap rows answer for, 1059 and 963
      // (merging every list: 1407).
      const uint32_t y = lane < d ? sm.list[lane] : 0u;
      const bool row_of = lane > 0 && lane < d;
      const uint4 b = row_of ? bit_row(a, y) : make_uint4(0, 0, 0, 0);
      const uint64_t e0 = row_of ? a.off[y] : 0ull, xe = row_of ? a.off[y + 1] : 0ull;
      uint32_t row = 0;
      for (uint32_t has = __ballot_sync(KCL_FULL, row_of && b.x != kNoBitRow); has; has &= has - 1) {
        const int i = __ffs((int)has) - 1;
        const uint32_t bo = __shfl_sync(KCL_FULL, b.x, i), bf = __shfl_sync(KCL_FULL, b.y, i);
        const uint32_t bs = __shfl_sync(KCL_FULL, b.z, i);
        const uint32_t m = __ballot_sync(KCL_FULL, lane < i && bit_at(a, bo, bf, bs, y));
        if (lane == i) row = m;
      }
      if (row_of && b.x == kNoBitRow) {
        int j = 0;
        uint32_t at = sm.list[0];
        for (uint64_t e = e0; e < xe && j < lane; e += 4) {
          uint32_t z[4];
#pragma unroll
          for (int q = 0; q < 4; ++q) z[q] = e + q < xe ? a.cols[e + q] : 0xffffffffu;
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            while (j < lane && at < z[q]) at = sm.list[++j];
            if (j < lane && at == z[q]) row |= 1u << j;
          }
        }
      }
      if constexpr (MODE == MODE_SEQ) {
        if (lane < d) sm.rows[lane] = row;
      } else {
        uint32_t full = row;  // symmetric: the column off the others' rows
        for (int g = 1; g < d; ++g) {
          const uint32_t m = __shfl_sync(KCL_FULL, row, g);
          if (lane < g && ((m >> lane) & 1u)) full |= 1u << g;
        }
        if constexpr (MODE == MODE_ORDER) {  // by key rank, upward
          uint32_t up = 0;
          for (uint32_t it = __shfl_sync(KCL_FULL, full, lane < d ? sm.inv[lane] : 0); it; it &= it - 1)
            up |= 1u << sm.rank[__ffs((int)it) - 1];
          full = lane < d ? up & ~((2u << lane) - 1u) : 0u;
        }
        if (lane < d) sm.rows[lane] = full;
      }
      __syncwarp();
    } else if (K >= 3) {
      // Row i: out-neighbours of list[i] inside N+(s) (MakeSubgraph's induced
      // adjacency, :104-113).  A member with a bitmap row is asked about every
      // member before it at once, a lane each; the others' out-lists are
      // walked, a lane per row.
      const uint32_t y0 = lane < d ? sm.list[lane] : 0u, y1 = lane + 32 < d ? sm.list[lane + 32] : 0u;
      const uint4 b0 = lane < d ? bit_row(a, y0) : make_uint4(0, 0, 0, 0);
      const uint4 b1 = lane + 32 < d ? bit_row(a, y1) : make_uint4(0, 0, 0, 0);
#pragma unroll 4
      for (int i = 1; i < d; ++i) {
        const uint32_t bo = __shfl_sync(KCL_FULL, i < 32 ? b0.x : b1.x, i & 31);
        const uint32_t bf = __shfl_sync(KCL_FULL, i < 32 ? b0.y : b1.y, i & 31);
        const uint32_t bs = __shfl_sync(KCL_FULL, i < 32 ? b0.z : b1.z, i & 31);  // 0: no row, no hit
        const bool h0 = lane < i && bit_at(a, bo, bf, bs, y0);
        const bool h1 = lane + 32 < i && bit_at(a, bo, bf, bs, y1);
        const uint32_t m0 = __ballot_sync(KCL_FULL, h0);
        const uint32_t m1 = i > 32 ? __ballot_sync(KCL_FULL, h1) : 0u;
        if (lane == 0) sm.rows[i] = (unsigned long long)m1 << 32 | m0;
      }
      const bool w0 = lane < d && b0.x == kNoBitRow, w1 = lane + 32 < d && b1.x == kNoBitRow;
      if (__any_sync(KCL_FULL, w0 || w1)) {
        const int tb = tab_bits((uint32_t)d);
        for (int i = lane; i < 1 << tb; i += 32) sm.tab[i] = kTabEmpty;
        __syncwarp();
        for (int i = lane; i < d; i += 32) tab_insert(sm.tab, tb, sm.list[i], i);
        __syncwarp();
        for (int i = lane; i < d; i += 32) {
          if (!(i < 32 ? w0 : w1) || i == 0) continue;
          const uint32_t x = sm.list[i], top = sm.list[i - 1];
          const uint64_t xe = a.off[x + 1];
          unsigned long long row = 0;
          for (uint64_t e = a.off[x]; e < xe; e += 4) {
            uint32_t y[4];
#pragma unroll
            for (int b = 0; b < 4; ++b) y[b] = e + b < xe ? a.cols[e + b] : 0xffffffffu;
#pragma unroll
            for (int b = 0; b < 4; ++b)
              if (y[b] <= top) {
                const int j = tab_find(sm.tab, tb, sm.list, y[b]);
                if (j >= 0) row |= 1ull << j;
              }
            if (y[3] > top) break;  // ascending: no later neighbour is in list[0, i)
          }
          sm.rows[i] = row;
        }
      }
      __syncwarp();
      if constexpr (MODE != MODE_SEQ) {
        // COUNT: symmetric rows; ORDER: rows by key rank, upward.  A lane reads
        // its whole row off the lower triangle: no bit is set by an atomic
        // (lanes meeting in a word made the former scatter the kernel's
        // longest phase, 228 us of a 64-member root's 245).
        const uint32_t *half = reinterpret_cast<const uint32_t *>(sm.rows);
        unsigned long long full[2] = {0, 0};
#pragma unroll
        for (int q = 0; q < 2; ++q) {
          const int p = lane + 32 * q;
          if (32 * q >= d) break;
          const int i = MODE == MODE_ORDER ? (p < d ? sm.inv[p] : 0) : p;
          uint32_t w[2] = {0, 0};
#pragma unroll
          for (int z = 0; z < 2; ++z) {
            if (MODE == MODE_ORDER && z < q) continue;  // upward: higher ranks only
            const int end = d - 32 * z < 32 ? d - 32 * z : 32;
            for (int b = 0; b < end; ++b) {
              const int j = MODE == MODE_ORDER ? sm.inv[32 * z + b] : 32 * z + b;
              const int hi = MODE == MODE_ORDER && i > j ? i : j, lo = MODE == MODE_ORDER && i > j ? j : i;
              if ((half[2 * hi + (lo >> 5)] >> (lo & 31)) & 1u) w[z] |= 1u << b;  // rows hold bits below their own
            }
          }
          full[q] = (unsigned long long)w[1] << 32 | w[0];
          if constexpr (MODE == MODE_ORDER) full[q] &= ~((2ull << p) - 1ull);
          else full[q] |= p < d ? sm.rows[p] : 0ull;
        }
        __syncwarp();
#pragma unroll
        for (int q = 0; q < 2; ++q)
          if (lane + 32 * q < d) sm.rows[lane + 32 * q] = full[q];
      }
      __syncwarp();
    }
    if constexpr (MODE == MODE_SEQ) {
      uint32_t *dl = &sm.dl[lane * kSDl];
      for (int j = lane; j < d; j += 32) {
        const unsigned long long C = sm.rows[j];
        if (!C) continue;
        const int g0 = sm.base[j] < sm.base[d] ? j : d;  // kCDensestNoAtom.c:287
        seq64<K - 2>(C, g0, sm.rows, sm.base, dl);
        // Close the stream: its increments fell on {s, t} ∪ C (shared loads:
        // straight to the load vector).
        auto close = [&](int i) {
          if (!dl[i]) return;
          if (a.shared_loads) atomicAdd(a.out + (i < d ? sm.list[i] : s), (unsigned long long)dl[i]);
          else shared_add(&sm.acc[i], dl[i]);
          dl[i] = 0;
        };
        unsigned long long it = C;
        while (it) {
          const int i = __ffsll((long long)it) - 1;
          it &= it - 1;
          close(i);
        }
        close(j);
        close(d);
      }
      __syncwarp();
      for (int i = lane; i <= d; i += 32) {
        const unsigned long long v = sm.acc[i];
        if (v) {
          atomicAdd(&a.out[i < d ? sm.list[i] : s], v);
          sm.acc[i] = 0;
        }
      }
    } else if constexpr (MODE == MODE_ORDER) {
      uint64_t ssum = 0;
      for (int p = lane; p < d; p += 32) {
        const uint64_t c = cnt64<K - 2, false>(sm.rows[p], sm.rows);
        if (p < tau) {
          if (c) atomicAdd(&a.out[sm.list[sm.inv[p]]], (unsigned long long)c);
        } else {
          ssum += c;
        }
      }
      ssum = warp_sum(ssum);
      if (lane == 0 && ssum) atomicAdd(&a.out[s], (unsigned long long)ssum);
    } else {
      uint64_t tot = 0;
      for (int x = lane; x < d; x += 32) {
        const uint64_t c = cnt64<K - 2, true>(sm.rows[x], sm.rows);
        if (a.list_off) a.pair_out[o + x] = (unsigned long long)c;
        else if (c) atomicAdd(&a.out[sm.list[x]], (unsigned long long)c);
        tot += c;
      }
      tot = warp_sum(tot);
      if (lane == 0 && tot && !a.list_off) {
        atomicAdd(&a.out[s], (unsigned long long)(tot / (K - 1)));
        if constexpr (IDENT) atomicAdd(a.total, (unsigned long long)(tot / (K - 1)));
      }
    }
    __syncwarp();
  }
}

// ========================================================================
// Tiers M and L: one CTA per root, rows of W 32-bit words, lane w holds word
// w (tier M, W <= 32) or words w and w + 32 (tier L, W <= 64).
template <int WPL>
struct Bits {
  uint32_t w[WPL];
};

// Seq rows hold only the ids below their own (N+(x) lies below x): row i
// keeps (i >> 5) + 1 words, packed one after another from word tri_off(i),
// which halves the bitmap and leaves shared memory for more stream warps.
__host__ __device__ __forceinline__ uint32_t tri_off(uint32_t i) {
  const uint32_t a = i >> 5, b = i & 31;
  return i + a * (16u * a + b - 16u * (a > 0));
}
template <int WPL, bool TRI = false>
__device__ __forceinline__ Bits<WPL> load_row(const uint32_t *rows, int r, int W, int lane) {
  Bits<WPL> b;
  const size_t o = TRI ? (size_t)tri_off((uint32_t)r) : (size_t)r * W;
  const int n = TRI ? (r >> 5) + 1 : W;
#pragma unroll
  for (int q = 0; q < WPL; ++q) {
    const int w = lane + 32 * q;
    b.w[q] = w < n ? rows[o + w] : 0u;
  }
  return b;
}
template <int WPL>
__device__ __forceinline__ Bits<WPL> band(const Bits<WPL> &a, const Bits<WPL> &b) {
  Bits<WPL> c;
#pragma unroll
  for (int q = 0; q < WPL; ++q) c.w[q] = a.w[q] & b.w[q];
  return c;
}
template <int WPL>
__device__ __forceinline__ int popc_lane(const Bits<WPL> &a) {
  int c = 0;
#pragma unroll
  for (int q = 0; q < WPL; ++q) c += __popc(a.w[q]);
  return c;
}
template <int WPL>
__device__ __forceinline__ bool any_bits(const Bits<WPL> &a) {
  uint32_t o = 0;
#pragma unroll
  for (int q = 0; q < WPL; ++q) o |= a.w[q];
  return __any_sync(KCL_FULL, o != 0);
}
// Mask of the ids below y for this lane's words.
template <int WPL>
__device__ __forceinline__ Bits<WPL> below_mask(int y, int lane) {
  Bits<WPL> b;
#pragma unroll
  for (int q = 0; q < WPL; ++q) {
    const int w = lane + 32 * q;
    const int yw = y >> 5;
    b.w[q] = w < yw ? 0xffffffffu : (w == yw ? ((1u << (y & 31)) - 1u) : 0u);
  }
  return b;
}

// Visit the members of a distributed set in ascending order (uniform across
// the warp).  F(u) is called by all lanes.
template <int WPL, typename F>
__device__ __forceinline__ void for_each_bit(const Bits<WPL> &P, F &&f) {
#pragma unroll
  for (int q = 0; q < WPL; ++q) {
    uint32_t m = __ballot_sync(KCL_FULL, P.w[q] != 0);
    while (m) {
      const int L = __ffs(m) - 1;
      m &= m - 1;
      uint32_t wb = __shfl_sync(KCL_FULL, P.w[q], L);
      while (wb) {
        const int b = __ffs(wb) - 1;
        wb &= wb - 1;
        f((L + 32 * q) * 32 + b);
      }
    }
  }
}

// Per-lane partial count of R-cliques inside P.
template <int R, bool BELOW, int WPL>
__device__ __forceinline__ uint64_t cnt_warp(const Bits<WPL> &P, const uint32_t *rows, int W, int lane) {
  if constexpr (R == 0) {
    return lane == 0 ? 1u : 0u;
  } else if constexpr (R == 1) {
    return (uint64_t)popc_lane(P);
  } else {
    uint64_t c = 0;
    for_each_bit<WPL>(P, [&](int y) {
      Bits<WPL> A = load_row<WPL>(rows, y, W, lane);
      if (BELOW) A = band(A, below_mask<WPL>(y, lane));
      c += cnt_warp<R - 1, BELOW, WPL>(band(P, A), rows, W, lane);
    });
    return c;
  }
}

// Edges of G_s inside P, each once, as per-lane partial sums (the k = 4 count,
// (k-2)-cliques = edges): the counting rows are symmetric and each member y
// counts its neighbours below it (BELOW), the Order rows are oriented upward
// and y counts its whole row.  P's members are compacted and a lane takes one
// member at a time, walking only the words its row can occupy -- instead of
// a warp per member over all W words (cnt_warp), which leaves the lanes past
// W idle and re-reads the empty half of every row.  scratch: 32 words for P,
// then the member list (u16).
template <bool BELOW>
__device__ __forceinline__ uint32_t edges_in(const Bits<1> &P, const uint32_t *rows, int W, int lane,
                                             uint32_t *scratch) {
  uint16_t *members = reinterpret_cast<uint16_t *>(scratch + 32);
  if (lane < W) scratch[lane] = P.w[0];
  const uint32_t lt = lanemask_lt();
  uint32_t total = 0;
  uint32_t nz = __ballot_sync(KCL_FULL, P.w[0] != 0);
  while (nz) {
    const int L = __ffs(nz) - 1;
    nz &= nz - 1;
    const uint32_t word = __shfl_sync(KCL_FULL, P.w[0], L);
    if ((word >> lane) & 1u) members[total + __popc(word & lt)] = (uint16_t)((L << 5) | lane);
    total += (uint32_t)__popc(word);
  }
  __syncwarp();
  uint32_t c = 0;
  for (uint32_t i = lane; i < total; i += 32) {
    const int y = members[i];
    const uint32_t *ry = rows + (size_t)y * W;
    if constexpr (BELOW) {
      const int hi = y >> 5;
      for (int w = 0; w < hi; ++w) c += __popc(scratch[w] & ry[w]);
      c += __popc(scratch[hi] & ry[hi] & ((1u << (y & 31)) - 1u));
    } else {
      for (int w = y >> 5; w < W; ++w) c += __popc(scratch[w] & ry[w]);
    }
  }
  __syncwarp();  // the next row reuses the scratch
  return c;
}

// Triangles of G_s inside P, each once, as per-lane partial sums (the k = 5
// count): a lane per member y of P walks the members z of P ∩ row(y) (below y
// with BELOW) and adds |P ∩ row(y) ∩ row(z)| over the words those rows can
// occupy.  scratch: cbuf_words(5, .) words.
template <bool BELOW>
__device__ __forceinline__ uint32_t triangles_in(const Bits<1> &P, const uint32_t *rows, int W, int lane,
                                                 uint32_t *scratch) {
  constexpr int cbuf_rows_at = 32;  // 64 rows of 64 bits, then the members
  uint16_t *members = reinterpret_cast<uint16_t *>(scratch + 32 + 128);
  if (lane < W) scratch[lane] = P.w[0];
  const uint32_t lt = lanemask_lt();
  uint32_t total = 0;
  uint32_t nz = __ballot_sync(KCL_FULL, P.w[0] != 0);
  while (nz) {
    const int L = __ffs(nz) - 1;
    nz &= nz - 1;
    const uint32_t word = __shfl_sync(KCL_FULL, P.w[0], L);
    if ((word >> lane) & 1u) members[total + __popc(word & lt)] = (uint16_t)((L << 5) | lane);
    total += (uint32_t)__popc(word);
  }
  __syncwarp();
  uint32_t c = 0;
  if (total <= 64) {
    // The rows among the members, as 64-bit masks: a step down the clique is
    // then one word, where the rows as they stand are walked over all words
    // they can occupy (a k = 5 Sim pass over RMAT-15 with planted communities,
    // members mostly 20..50: 725 -> 658 us).
    unsigned long long *R = reinterpret_cast<unsigned long long *>(scratch + cbuf_rows_at);
    const uint32_t m0 = lane < total ? members[lane] : 0u, m1 = lane + 32 < total ? members[lane + 32] : 0u;
    const uint32_t *col0 = rows + (m0 >> 5), *col1 = rows + (m1 >> 5);
    const uint32_t bit0 = lane < total ? 1u << (m0 & 31) : 0u, bit1 = lane + 32 < total ? 1u << (m1 & 31) : 0u;
    unsigned long long mine[2] = {0, 0};
    for (uint32_t g = 0; g < total; ++g) {
      const uint32_t o = (uint32_t)members[g] * (uint32_t)W;
      const uint32_t b0 = __ballot_sync(KCL_FULL, (col0[o] & bit0) != 0);
      const uint32_t b1 = total > 32 ? __ballot_sync(KCL_FULL, (col1[o] & bit1) != 0) : 0u;
      const unsigned long long row = ((unsigned long long)b1 << 32 | b0) & (BELOW ? (1ull << g) - 1ull : ~0ull);
      if (lane == (int)(g & 31u)) {
        if (g < 32) mine[0] = row;
        else mine[1] = row;
        R[g] = row;
      }
    }
    __syncwarp();
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      const unsigned long long r = mine[q];
      for (unsigned long long it = r; it; it &= it - 1) c += (uint32_t)__popcll(r & R[__ffsll((long long)it) - 1]);
    }
    __syncwarp();  // the next row reuses the scratch
    return c;
  }
  for (uint32_t i = lane; i < total; i += 32) {
    const int y = members[i];
    const uint32_t *ry = rows + (size_t)y * W;
    const int lo_w = BELOW ? 0 : (y >> 5), hi_w = BELOW ? (y >> 5) : W - 1;
    for (int w = lo_w; w <= hi_w; ++w) {
      uint32_t q = scratch[w] & ry[w];
      if (BELOW && w == (y >> 5)) q &= (1u << (y & 31)) - 1u;
      while (q) {
        const int b = __ffs(q) - 1;
        q &= q - 1;
        const int z = (w << 5) | b;
        const uint32_t *rz = rows + (size_t)z * W;
        if constexpr (BELOW) {
          const int zh = z >> 5;
          for (int w2 = 0; w2 < zh; ++w2) c += __popc(scratch[w2] & ry[w2] & rz[w2]);
          c += __popc(scratch[zh] & ry[zh] & rz[zh] & ((1u << (z & 31)) - 1u));
        } else {
          for (int w2 = z >> 5; w2 < W; ++w2) c += __popc(scratch[w2] & ry[w2] & rz[w2]);
        }
      }
    }
  }
  __syncwarp();  // the next row reuses the scratch
  return c;
}

constexpr int kPairMembers = 256;  // most members of PairLevel's I
// Words of PairLevel's per-warp scratch: P's words, a group's row offsets and (value,
// range) pairs, I's values, increments and positions, the members of P.
__host__ __device__ inline size_t pair_words(uint32_t dmax) {
  return 32 + 32 + 64 + kPairMembers + kPairMembers / 4 + kPairMembers / 2 + (((size_t)dmax + 7) / 8) * 4;
}

// Words of a Seq warp: the stream's values or increments (dmax + 1), and with
// rows in shared memory at k >= 4 the last two levels' scratch.  At k = 4 a
// stream uses one or the other, so they share the words.
__host__ __device__ inline size_t seq_warp_words(int k, uint32_t dmax, bool rows_in_smem) {
  const size_t v = ((size_t)dmax + 4) / 4 * 4, p = k >= 4 && rows_in_smem ? pair_words(dmax) : 0;
  return k == 4 ? (v > p ? v : p) : v + p;
}
// Shared-memory layout of a tier M / L CTA (dmax = largest out-degree the
// launch allows, NW warps).  Tier L keeps `rows` in a global slab instead.
struct LayoutM {
  size_t list, tab, rows, base, acc, rel, rank, inv, dl, cbuf, total;
};
// Per-warp scratch of the k = 4, 5 counting paths: P's words, (k = 5) the rows
// among 64 members, and P's members, compacted.
__host__ __device__ inline size_t cbuf_words(int k, uint32_t dmax) {
  return (32 + (k == 5 ? 128 : 0) + ((size_t)dmax + 1) / 2 + 3) / 4 * 4;
}
__host__ __device__ inline size_t align16(size_t x) { return (x + 15) & ~(size_t)15; }
__host__ __device__ inline LayoutM layout_m(int mode, int k, uint32_t dmax, int nw, bool rows_in_smem) {
  LayoutM L;
  const size_t W = (dmax + 31) / 32;
  size_t at = 0;
  L.list = at; at = align16(at + (size_t)dmax * 4);
  L.tab = at; at = align16(at + ((size_t)4 << tab_bits(dmax)));
  L.rows = at;
  if (rows_in_smem) at = align16(at + (mode == MODE_SEQ ? (size_t)tri_off(dmax) : (size_t)dmax * W) * 4);
  L.base = at; if (mode != MODE_COUNT) at = align16(at + (size_t)(dmax + 1) * 8);
  L.acc = at; if (mode == MODE_SEQ) at = align16(at + (size_t)(dmax + 1) * 8);
  L.rank = at; if (mode == MODE_ORDER) at = align16(at + (size_t)dmax * 2);
  L.inv = at; if (mode == MODE_ORDER) at = align16(at + (size_t)dmax * 2);
  L.rel = at; if (mode == MODE_SEQ && rows_in_smem) at = align16(at + (size_t)(dmax + 1) * 4);
  L.dl = at; if (mode == MODE_SEQ) at = align16(at + (size_t)nw * seq_warp_words(k, dmax, rows_in_smem) * 4);
  L.cbuf = at;
  if (mode != MODE_SEQ && (k == 4 || k == 5) && rows_in_smem) at = align16(at + (size_t)nw * cbuf_words(k, dmax) * 4);
  L.total = at;
  return L;
}

// Current values of a root-edge stream's vertices (pass-start r plus the
// stream's own increments), in one of two forms:
//  * Vals32: one u32 per vertex, offset from the smallest pass-start value of
//    the stream (off) and capped at cap, when every value the stream can reach
//    stays below 2^31 (see seq_stream);
//  * Vals64: the pass-start u64 plus a u32 delta per vertex.
// Vertex x's word is only ever read and written by lane x & 31 (the chain,
// the argmin write-backs, the stream's setup and close), so the chains need
// no warp barrier.
struct Vals32 {
  using T = uint32_t;
  uint32_t *cur;
  __device__ __forceinline__ T get(int v, uint32_t &raw) const { raw = cur[v]; return raw; }
  __device__ __forceinline__ void bump(int v, uint32_t raw, uint32_t *) const { cur[v] = raw + 1u; }
  __device__ __forceinline__ void add(int v, T delta, uint32_t *) const { cur[v] += delta; }
};
template <bool OVF>
struct Vals64 {
  using T = unsigned long long;
  const unsigned long long *base;
  uint32_t *dl;
  __device__ __forceinline__ T get(int v, uint32_t &raw) const { raw = dl[v]; return base[v] + raw; }
  __device__ __forceinline__ void bump(int v, uint32_t raw, uint32_t *err) const {
    if (OVF && raw == 0xffffffffu) atomicOr(err, ERR_OVERFLOW);
    dl[v] = raw + 1u;
  }
  __device__ __forceinline__ void add(int v, T delta, uint32_t *err) const {
    const unsigned long long nd = (unsigned long long)dl[v] + delta;
    if (OVF && nd > 0xffffffffull) atomicOr(err, ERR_OVERFLOW);
    dl[v] = (uint32_t)nd;
  }
};

// Shared loads (KCLPP_SEQ_SHARED): a vertex's current value is the CTA's copy
// of the pass's one load vector -- 32 bits, relative to the smallest value
// of the root's vertices when the root started, capped at kSharedCap --
// refreshed from the vector when a stream starts and raised by the CTA's
// closing streams, plus this stream's own increments (a u32 per vertex, owned
// by lane v & 31 as in Vals64).  Other warps refresh and close concurrently,
// so a read is a recent snapshot, and a capped value hides how far above the
// others it is: the values steer which member gets a unit, never whether a
// unit is given.
constexpr uint32_t kSharedCap = 1u << 29;
struct ValsShared {
  using T = uint32_t;
  const uint32_t *cur;
  uint32_t *dl;
  __device__ __forceinline__ T get(int v, uint32_t &raw) const {
    raw = dl[v];
    return *(const volatile uint32_t *)(cur + v) + raw;
  }
  __device__ __forceinline__ void bump(int v, uint32_t raw, uint32_t *err) const {
    if (raw == 0xffffffffu) atomicOr(err, ERR_OVERFLOW);
    dl[v] = raw + 1u;
  }
  __device__ __forceinline__ void add(int v, T delta, uint32_t *err) const {
    const unsigned long long nd = (unsigned long long)dl[v] + delta;
    if (nd > 0xffffffffull) atomicOr(err, ERR_OVERFLOW);
    dl[v] = (uint32_t)nd;
  }
};

// Distance from the prefix value c to a candidate's value, as the chain's
// fixed point uses it: -1 below c, else the difference clamped to 2^31 - 1
// (a plain 32-bit difference for Vals32, whose values all lie below 2^31).
template <typename T>
__device__ __forceinline__ int distance(T av, T c) {
  if constexpr (sizeof(T) == 4) {
    return (int)(av - c);
  } else {
    if (av < c) return -1;
    const T dd = av - c;
    return dd > 0x7fffffffull ? 0x7fffffff : (int)dd;
  }
}

// The fixed point of one 32-candidate word of the chain: lane b stands for
// candidate b of the word (valid when its bit is set), rel its distance to
// the prefix value c at the word's start.  Candidate i falls to the prefix
// iff rel_i >= the number of earlier candidates of the word that fell to it
// (kCDensestNoAtom.c:162-171 and 180-186, resolved by ballots).  Returns the
// mask of the candidates that fall.
__device__ __forceinline__ uint32_t word_fixed_point(int rel, uint32_t lt) {
  // Start from "every candidate at or above c falls": once the loads have
  // spread, that guess is already exact and one vote confirms it; ties (the
  // first pass) take a few more rounds.  When no candidate is at or above c,
  // every one takes its clique and the guess is the fixed point already.
  uint32_t m = __ballot_sync(KCL_FULL, rel >= 0);
  if (m) {
    uint32_t m2 = __ballot_sync(KCL_FULL, rel >= __popc(m & lt));
    if (m2 != m) {
      m = m2;
      for (int r = 0; r < 32; ++r) {
        m2 = __ballot_sync(KCL_FULL, rel >= __popc(m & lt));
        if (m2 == m) break;
        m = m2;
      }
    }
  }
  return m;
}

// The Seq chain over V (the last level), one 32-bit word of V at a time: lane
// b stands for candidate 32 * word + b.  c is the current value of the prefix
// argmin (kCDensestNoAtom.c:162-171 and 180-186: each clique goes to the
// candidate w when r[w] < c, strict, else to the prefix argmin, whose value
// then grows by one).  Returns the prefix argmin's new value.
template <int WPL, typename VA>
__device__ __forceinline__ typename VA::T chain_words(const Bits<WPL> &V, typename VA::T c, const VA &va, int lane,
                                                      uint32_t *err) {
  using T = typename VA::T;
  const uint32_t lt = lanemask_lt();
#pragma unroll
  for (int q = 0; q < WPL; ++q) {
    uint32_t nz = __ballot_sync(KCL_FULL, V.w[q] != 0);
    while (nz) {
      const int L = __ffs(nz) - 1;
      nz &= nz - 1;
      const uint32_t word = __shfl_sync(KCL_FULL, V.w[q], L);
      const bool valid = (word >> lane) & 1u;
      const int v = ((L + 32 * q) << 5) | lane;
      int rel = -1;
      uint32_t raw = 0;
      if (valid) rel = distance<T>(va.get(v, raw), c);
      const uint32_t m = word_fixed_point(rel, lt);
      if (valid && !((m >> lane) & 1u)) va.bump(v, raw, err);
      c += (T)__popc(m);
    }
  }
  return c;
}

// The same chain over V of one word per lane (lane w holds word w of V) with
// 32-bit values, skipping the words that fall whole.  lo (lane w): the
// smallest value the stream started with among C's members in word w.
// Values only grow, and the prefix value at any candidate of V is at most c
// plus the number of candidates before it (< tot), so every candidate of a
// word with lo >= c + tot - 1 falls to the prefix: only the other words run
// their fixed point, in order, each from its exact prefix value c + (the
// candidates of V before it) - (those of them that took their clique).
template <typename VA>
__device__ __forceinline__ uint32_t chain_word1(uint32_t q, uint32_t c, const VA &va, uint32_t lo, int lane,
                                                uint32_t *err) {
  const uint32_t pop = (uint32_t)__popc(q);
  const uint32_t tot = __reduce_add_sync(KCL_FULL, pop);
  if (!tot) return c;
  uint32_t bad = __ballot_sync(KCL_FULL, pop != 0u && lo < c + tot - 1u);
  if (!bad) return c + tot;
  const uint32_t lt = lanemask_lt();
  uint32_t taken = 0;
  do {
    const int L = __ffs(bad) - 1;
    bad &= bad - 1;
    const uint32_t before = __reduce_add_sync(KCL_FULL, lane < L ? pop : 0u);
    const uint32_t cL = c + before - taken;
    const uint32_t word = __shfl_sync(KCL_FULL, q, L);
    const bool valid = (word >> lane) & 1u;
    const int v = (L << 5) | lane;
    int rel = -1;
    uint32_t raw = 0;
    if (valid) rel = (int)(va.get(v, raw) - cL);
    const uint32_t m = word_fixed_point(rel, lt);
    if (valid && !((m >> lane) & 1u)) va.bump(v, raw, err);
    taken += (uint32_t)(__popc(word) - __popc(m));
  } while (bad);
  return c + tot - taken;
}

// Current value of vertex x, read by the lane that owns it and broadcast.
template <typename VA>
__device__ __forceinline__ typename VA::T value_of(int x, const VA &va, int lane) {
  typename VA::T v = 0;
  uint32_t raw;
  if ((x & 31) == lane) v = va.get(x, raw);
  return __shfl_sync(KCL_FULL, v, x & 31);
}

// Values of a root as 32-bit offsets from its smallest, capped here (the Seq
// kernel with rows in shared memory).
constexpr uint32_t kRelCap = 0x7ffffff0u;

// A whole stream over at most 32 * S candidates, in registers: member i of C
// is a bit of a mask and a lane (slot i >> 5), which keeps its value, its
// neighbours below it (crow) and above it (ccol).  Deeper prefixes are masks,
// so a level costs no set-up, and the last two levels are settled by counting
// or walked chain by chain as in PairLevel (whose ranges S_i are here exact
// counts: i's chances as a candidate and its own chain).  Streams of this size
// are all there is in sparse graphs: 24 Chung-Lu / Erdos-Renyi graphs at
// k = 3..7 take 12.9 ms for 2 passes with it, 19.6 ms with PairLevel for every
// stream, 25.2 ms with the word-at-a-time chain.
template <int S>
struct TinyStream {
  using M = typename std::conditional<S == 1, uint32_t, unsigned long long>::type;
  uint32_t v[S];
  M crow[S], ccol[S];
  int lane;

  static __device__ __forceinline__ int pop(M x) {
    if constexpr (S == 1) return __popc(x);
    else return __popcll(x);
  }
  static __device__ __forceinline__ int first(M x) {
    if constexpr (S == 1) return __ffs((int)x) - 1;
    else return __ffsll((long long)x) - 1;
  }
  // x[slot of u] from u's lane.
  template <typename T>
  __device__ __forceinline__ T of(const T (&x)[S], int u) const {
    T y = x[0];
    if constexpr (S == 2) y = u >= 32 ? x[1] : x[0];
    return __shfl_sync(KCL_FULL, y, u & 31);
  }
  static __device__ __forceinline__ M mask_of(const bool (&b)[S]) {
    M m = __ballot_sync(KCL_FULL, b[0]);
    if constexpr (S == 2) m |= (M)__ballot_sync(KCL_FULL, b[1]) << 32;
    return m;
  }
  __device__ __forceinline__ bool in(M x, int q) const { return (x >> (32 * q + lane)) & 1u; }

  // list: C's members; the rows are read word by word, a lane per candidate.
  __device__ __forceinline__ void load(const uint32_t *rows, const uint16_t *list, int nc, const uint32_t *rel) {
    const uint32_t *col[S];
    uint32_t bit[S], off[S];
#pragma unroll
    for (int q = 0; q < S; ++q) {
      const int i = 32 * q + lane;
      const uint32_t id = i < nc ? list[i] : 0u;
      v[q] = i < nc ? rel[id] : kRelCap;
      col[q] = rows + (id >> 5);
      bit[q] = 1u << (id & 31);
      off[q] = tri_off(id);
      crow[q] = ccol[q] = 0;
    }
    for (int g = 1; g < nc; ++g) {
      const uint32_t o = of(off, g);
      bool has[S];
#pragma unroll
      for (int q = 0; q < S; ++q) {
        has[q] = 32 * q + lane < g && (col[q][o] & bit[q]);
        if (has[q]) ccol[q] |= (M)1 << g;
      }
      const M m = mask_of(has);
#pragma unroll
      for (int q = 0; q < S; ++q)
        if (32 * q + lane == g) crow[q] = m;
    }
  }

  __device__ __forceinline__ uint32_t pairs(M P, uint32_t c) {
    const uint32_t lt = lanemask_lt();
    uint32_t tot[S], R[S], mine = 0;
    bool act[S];
#pragma unroll
    for (int q = 0; q < S; ++q) {
      const bool here = in(P, q);
      tot[q] = here ? (uint32_t)pop(crow[q] & P) : 0u;
      R[q] = here ? (uint32_t)pop(ccol[q] & P) + tot[q] : 0u;
      act[q] = tot[q] != 0;
      mine += tot[q];
    }
    const uint32_t sum = __reduce_add_sync(KCL_FULL, mine);
    if (sum == 0) return c;
    bool low[S], amb = false;
#pragma unroll
    for (int q = 0; q < S; ++q) {
      low[q] = R[q] != 0 && v[q] + R[q] < c;
      amb |= R[q] != 0 && !low[q] && v[q] < c + sum;
    }
    if (!__any_sync(KCL_FULL, amb)) {
      const M Lg = mask_of(low);
      if (!Lg) return c + sum;
      uint32_t inc[S], taken = 0;
#pragma unroll
      for (int q = 0; q < S; ++q) {
        inc[q] = low[q] ? (uint32_t)pop(ccol[q] & P & ~Lg) : 0u;
        taken += inc[q];
      }
      bool clash = false;
      for (M rem = Lg & mask_of(act); rem; rem &= rem - 1) {
        const int u = first(rem);
        const uint32_t vu = of(v, u), ru = of(R, u);
        bool take[S];
#pragma unroll
        for (int q = 0; q < S; ++q) {
          const bool has = low[q] && ((ccol[q] >> u) & 1u);
          take[q] = has && v[q] + R[q] < vu;
          clash |= has && !take[q] && v[q] < vu + ru;
          inc[q] += take[q];
        }
        const uint32_t n = (uint32_t)pop(mask_of(take));
#pragma unroll
        for (int q = 0; q < S; ++q)
          if (32 * q + lane == u) inc[q] += tot[q] - n;
      }
      if (!__any_sync(KCL_FULL, clash)) {
        uint32_t fell = 0u - taken;
#pragma unroll
        for (int q = 0; q < S; ++q) {
          v[q] += inc[q];
          if (!low[q]) fell += tot[q];
        }
        return c + __reduce_add_sync(KCL_FULL, fell);
      }
    }
    // One chain after another, the u's of a slot at a time: those of the first
    // slot have candidates in it alone, and 32-bit masks serve.
#pragma unroll
    for (int z = 0; z < S; ++z) {
      for (uint32_t rem = __ballot_sync(KCL_FULL, act[z]); rem; rem &= rem - 1) {
        const int b = __ffs((int)rem) - 1;
        const uint32_t vu = __shfl_sync(KCL_FULL, v[z], b);
        const bool own = vu < c;  // strict: ties stay with the earlier argmin
        const uint32_t c0 = own ? vu : c;
        uint32_t c1 = c0;
#pragma unroll
        for (int q = 0; q <= z; ++q) {
          const uint32_t vm = __shfl_sync(KCL_FULL, (uint32_t)(crow[z] >> (32 * q)), b) & (uint32_t)(P >> (32 * q));
          if (z == 0 || vm) {
            const uint32_t m = word_fixed_point((vm >> lane) & 1u ? (int)(v[q] - c1) : -1, lt);
            v[q] += ((vm & ~m) >> lane) & 1u;
            c1 += (uint32_t)__popc(m);
          }
        }
        if (!own) c = c1;
        else if (lane == b) v[z] += c1 - c0;
      }
    }
    return c;
  }

  // Level L of the stream over P (kCDensestNoAtom.c:218-267).
  template <int L>
  __device__ __forceinline__ uint32_t level(M P, uint32_t c) {
    if constexpr (L == 2) {
      return pairs(P, c);
    } else {
      for (M rem = P; rem; rem &= rem - 1) {
        const int u = first(rem);
        const M Q = P & of(crow, u);
        if (pop(Q) < L - 1) continue;
        const uint32_t vu = of(v, u);
        const bool own = vu < c;
        const uint32_t c0 = own ? vu : c;
        const uint32_t c1 = level<L - 1>(Q, c0);
        if (own) {
#pragma unroll
          for (int q = 0; q < S; ++q)
            if (32 * q + lane == u) v[q] += c1 - c0;
        } else {
          c = c1;
        }
      }
      return c;
    }
  }

  template <int K>
  __device__ __forceinline__ uint32_t run(const uint32_t *rows, const uint16_t *list, int nc, const uint32_t *rel,
                                          unsigned long long *acc, uint32_t c) {
    load(rows, list, nc, rel);
    c = level<K - 2>(nc == 32 * S ? ~(M)0 : ((M)1 << nc) - 1, c);
#pragma unroll
    for (int q = 0; q < S; ++q) {
      const int i = 32 * q + lane;
      if (i < nc) {
        const uint32_t id = list[i], d = v[q] - rel[id];
        if (d) shared_add(acc + id, d);
      }
    }
    return c;
  }
};

// Bits over a group of ng rows (offsets ro[0..ng), 16-byte aligned, zero up to a
// multiple of 4; members [a, a + ng) of a list): bit g set iff the group's row
// g holds the member of local id `id` and list position j.  The rows are read
// word by word at its bit.  A row ends at its own word; what is read beyond
// belongs to ids above the row's and is masked off (only rows after j hold it).
__device__ __forceinline__ uint32_t column_bits(const uint32_t *rows, const uint32_t *ro, uint32_t id, int j, int a,
                                                int ng) {
  const uint32_t *col = rows + (id >> 5);
  const uint32_t bit = 1u << (id & 31);
  uint32_t t = 0;
  for (int g = 0; g < ng; g += 4) {
    const uint4 o = *reinterpret_cast<const uint4 *>(ro + g);
    uint32_t x = 0;
    if (col[o.x] & bit) x |= 1u;
    if (col[o.y] & bit) x |= 2u;
    if (col[o.z] & bit) x |= 4u;
    if (col[o.w] & bit) x |= 8u;
    t |= x << g;
  }
  const int lo = j + 1 - a;
  const uint32_t gmask = ng < 32 ? (1u << ng) - 1u : 0xffffffffu;
  return t & (lo <= 0 ? gmask : (lo >= 32 ? 0u : gmask & (0xffffffffu << lo)));
}

// The members of P (lane w: word w), ascending, into list.
__device__ __forceinline__ int list_members(uint32_t P, uint16_t *list, int lane) {
  const uint32_t lt = lanemask_lt();
  int np = 0;
  uint32_t nz = __ballot_sync(KCL_FULL, P != 0);
  while (nz) {
    const int L = __ffs(nz) - 1;
    nz &= nz - 1;
    const uint32_t word = __shfl_sync(KCL_FULL, P, L);
    if ((word >> lane) & 1u) list[np + __popc(word & lt)] = (uint16_t)((L << 5) | lane);
    np += __popc(word);
  }
  return np;
}

// The last two levels of a stream, at once: for u in P ascending, the chain
// over V = P ∩ row(u) (kCDensestNoAtom.c:173-188), values in 32 bits.
//
// What bounds these levels is instruction issue, and a walk over the words of
// every V spends it on lanes without a candidate and on candidates whose fate
// is known.  A member whose value is at or above c + |P| (|P| - 1) / 2 -- c
// plus every clique of the call -- can never be below a prefix value: it falls
// every time and never changes.  Only the others, I, are followed, compacted
// 32 to a slot.  The members u are taken 32 at a time (lane g: u_g, with
// tot_g = |V|).
//
// A group whose comparisons cannot change their outcome while it runs is
// settled by counting.  Inside the group i's value stays in [v_i, v_i + S_i],
// S_i = 32 + (i in the group: tot_i), and the prefix value in [c, c + sum
// tot].  If every i lies wholly below c (class L) or at or above c + sum tot,
// every chain of a u outside L gives its unit to exactly the members of V in
// L, the rest falls to the prefix; a u in L is its own prefix (value v_u, up
// to v_u + S_u) and is compared the same way with its V.  T_i, in i's lane,
// has bit g set iff i is in u_g's V, so these are popcounts.  When any two of
// the compared ranges overlap, the group's chains run one after another.
//
// Measured on a trimmed RMAT-18 core (233 K edges, k = 4, loads of 4 passes):
// 94 % of the groups settle; a pass 3.87 -> 1.47 ms against the word-at-a-time
// chain alone.  From zero, where nothing settles (k = 5, RMAT-15 with planted
// communities), 15.0 -> 11.9 ms.  At most 40 registers at k = 4 (48 warps per
// SM): at 80 (24 warps) the same pass took 2.16 ms.
//
// ACC: the values are the root's own (shared by its streams, read only) and
// increments go to acc; else the values are the stream's and are updated.
template <bool ACC>
struct PairLevel {
  const uint32_t *rows;     // the root's triangular rows
  uint32_t *val;            // values by local id
  unsigned long long *acc;  // ACC: the root's increments
  uint32_t *scratch;        // pair_words(dmax) words, 16-byte aligned
  int lane;

  __device__ __forceinline__ uint32_t *pw() const { return scratch; }
  __device__ __forceinline__ uint32_t *ro() const { return scratch + 32; }
  __device__ __forceinline__ uint2 *sv() const { return reinterpret_cast<uint2 *>(scratch + 64); }
  __device__ __forceinline__ uint32_t *vv() const { return scratch + 128; }
  __device__ __forceinline__ uint8_t *ci() const { return reinterpret_cast<uint8_t *>(scratch + 128 + kPairMembers); }
  __device__ __forceinline__ uint16_t *ilist() const {
    return reinterpret_cast<uint16_t *>(scratch + 128 + kPairMembers + kPairMembers / 4);
  }
  __device__ __forceinline__ uint16_t *list() const { return ilist() + kPairMembers; }

  // Lane g's row offset and tot: |P ∩ row(u)|.
  __device__ __forceinline__ uint32_t tot_of(int j, int np, uint32_t &off) const {
    uint32_t t = 0;
    off = 0;
    if (j < np) {
      const uint32_t u = list()[j];
      off = tri_off(u);
      const uint32_t *r = rows + off, *p = pw();
      const int hi = (int)(u >> 5);
      for (int w = 0; w <= hi; ++w) t += (uint32_t)__popc(r[w] & p[w]);
    }
    return t;
  }

  __device__ __forceinline__ void put(uint32_t id, uint32_t v0, uint32_t v) const {
    if constexpr (ACC) {
      if (v != v0) shared_add(acc + id, v - v0);
    } else {
      val[id] = v;
    }
  }

  // A chain of one slot whose every candidate is in I with nothing between
  // them: the takers among `has` from prefix value c (which grows by the rest).
  __device__ __forceinline__ uint32_t takers_dense(bool has, uint32_t v, uint32_t &c, uint32_t lt) const {
    const uint32_t vm = __ballot_sync(KCL_FULL, has);
    if (!vm) return 0;
    const uint32_t m = word_fixed_point(has ? (int)(v - c) : -1, lt);
    c += (uint32_t)__popc(m);
    return vm & ~m;
  }
  // The same when members outside I stand between them: `ahead` members of V
  // come before this lane's, of which `taken` took their clique in earlier
  // slots; a candidate takes iff its value is below c + ahead - (takers before).
  __device__ __forceinline__ uint32_t takers_sparse(bool has, uint32_t v, uint32_t c, uint32_t ahead, uint32_t taken,
                                                    uint32_t lt) const {
    const int z = has ? (int)(ahead + c - v - taken) : 0;
    uint32_t mk = __ballot_sync(KCL_FULL, z > 0);
    if (mk) {
      for (int it = 0; it < 33; ++it) {
        const uint32_t m2 = __ballot_sync(KCL_FULL, z > __popc(mk & lt));
        if (m2 == mk) break;
        mk = m2;
      }
    }
    return mk;
  }
  // V's words (lane = word) and the members of V in the words before it.
  __device__ __forceinline__ void words_of(uint32_t u, uint32_t off, uint32_t &Q, uint32_t &pre) const {
    Q = lane <= (int)(u >> 5) ? rows[off + lane] & pw()[lane] : 0u;
    const uint32_t own = (uint32_t)__popc(Q);
    pre = own;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t y = __shfl_up_sync(KCL_FULL, pre, o);
      if (lane >= o) pre += y;
    }
    pre -= own;
  }
  __device__ __forceinline__ uint32_t ahead_of(uint32_t id, uint32_t Q, uint32_t pre) const {
    const uint32_t w = __shfl_sync(KCL_FULL, Q, id >> 5), p = __shfl_sync(KCL_FULL, pre, id >> 5);
    return p + (uint32_t)__popc(w & ((1u << (id & 31)) - 1u));
  }

  // At most one slot: values in registers.  ALL: I is all of P (<= 32).
  template <bool ALL>
  __device__ __forceinline__ uint32_t run1(int np, int ni, uint32_t c) const {
    const uint32_t lt = lanemask_lt();
    const int at = lane < ni ? (ALL ? lane : (int)ilist()[lane]) : -1;
    const uint32_t id = at >= 0 ? list()[at] : 0u;
    const uint32_t v0 = at >= 0 ? val[id] : 0x7fffffffu;
    uint32_t v = v0;
    for (int a = 0; a < np; a += 32) {
      const int ng = np - a < 32 ? np - a : 32;
      uint32_t off;
      const uint32_t tot = tot_of(a + lane, np, off);
      const uint32_t sum = __reduce_add_sync(KCL_FULL, tot);
      if (sum == 0) continue;
      const int gi = at - a;
      const bool live = at >= 0 && gi < ng, in = live && gi >= 0;
      const uint32_t ti = __shfl_sync(KCL_FULL, tot, gi & 31);
      const uint32_t S = 32u + (in ? ti : 0u);
      const bool low = live && v + S < c;
      if (!__any_sync(KCL_FULL, live && !low && v < c + sum)) {
        if (!__any_sync(KCL_FULL, low)) {
          c += sum;
          continue;
        }
        const uint32_t Lg = __reduce_or_sync(KCL_FULL, in && low ? 1u << gi : 0u);
        __syncwarp();
        ro()[lane] = off;
        if (in && low) sv()[gi] = make_uint2(v, S);
        __syncwarp();
        uint32_t T = column_bits(rows, ro(), id, at, a, ng);
        if (!low) T = 0;  // the others always fall
        uint32_t inc = (uint32_t)__popc(T & ~Lg);
        const uint32_t taken = inc;
        bool clash = false;
        for (uint32_t rem = Lg; rem; rem &= rem - 1) {
          const int g = __ffs(rem) - 1;
          const uint2 x = sv()[g];
          const bool has = (T >> g) & 1u, take = has && v + S < x.x;
          clash |= has && !take && v < x.x + x.y;
          const uint32_t n = (uint32_t)__popc(__ballot_sync(KCL_FULL, take));
          inc += take;
          if (in && gi == g) inc += ti - n;
        }
        if (!__any_sync(KCL_FULL, clash)) {
          v += inc;
          c += __reduce_add_sync(KCL_FULL, (((Lg >> lane) & 1u) ? 0u : tot) - taken);
          continue;
        }
      }
      const uint32_t *col = rows + (id >> 5);
      const uint32_t bit = 1u << (id & 31);
      for (uint32_t rem = __ballot_sync(KCL_FULL, tot != 0); rem; rem &= rem - 1) {
        const int g = __ffs(rem) - 1;
        const uint32_t og = __shfl_sync(KCL_FULL, off, g);
        const bool has = at >= 0 && gi < g && (col[og] & bit);
        uint32_t vu = 0x7fffffffu;
        if constexpr (ALL) {
          vu = __shfl_sync(KCL_FULL, v, g);
        } else {
          const uint32_t who = __ballot_sync(KCL_FULL, in && gi == g);
          if (who) vu = __shfl_sync(KCL_FULL, v, __ffs(who) - 1);
        }
        const bool own = vu < c;  // strict: ties stay with the earlier argmin
        const uint32_t c0 = own ? vu : c;
        uint32_t fell, mk;
        if constexpr (ALL) {
          uint32_t cl = c0;
          mk = takers_dense(has, v, cl, lt);
          fell = cl - c0;
        } else {
          const uint32_t tu = __shfl_sync(KCL_FULL, tot, g);
          const uint32_t x = v - c0;
          if (!__any_sync(KCL_FULL, has && x < tu)) {
            mk = __ballot_sync(KCL_FULL, has && (int)x < 0);
          } else {
            uint32_t Q, pre;
            words_of(list()[a + g], og, Q, pre);
            mk = takers_sparse(has, v, c0, ahead_of(id, Q, pre), 0u, lt);
          }
          fell = tu - (uint32_t)__popc(mk);
        }
        v += (mk >> lane) & 1u;
        if (!own) c += fell;
        else if (in && gi == g) v += fell;
      }
    }
    if (at >= 0) put(id, v0, v);
    __syncwarp();
    return c;
  }

  // Several slots: values, increments and positions in the scratch, member
  // 32 q + lane of I always handled by this lane.
  __device__ __forceinline__ uint32_t run_slots(int np, int ni, uint32_t c) const {
    const uint32_t lt = lanemask_lt();
    const bool dense = ni == np;
    uint32_t *const V = vv();
    uint8_t *const I8 = ci();
    const uint16_t *const il = ilist();
    for (int i = lane; i < ni; i += 32) V[i] = val[list()[il[i]]];
    for (int a = 0; a < np; a += 32) {
      const int ng = np - a < 32 ? np - a : 32;
      uint32_t off;
      const uint32_t tot = tot_of(a + lane, np, off);
      const uint32_t sum = __reduce_add_sync(KCL_FULL, tot);
      if (sum == 0) continue;
      int ns = 0;  // slots with a member at or before the group's last
      while (32 * ns < ni && (int)il[32 * ns] < a + ng) ++ns;
      uint32_t Lg = 0, Ig = 0;
      bool amb = false, lows = false;
      __syncwarp();
      ro()[lane] = off;
      for (int q = 0; q < ns; ++q) {
        const int i = 32 * q + lane;
        const int gi = i < ni ? (int)il[i] - a : 64;
        const bool live = gi < ng, in = live && gi >= 0;
        const uint32_t ti = __shfl_sync(KCL_FULL, tot, gi & 31);
        if (live) {
          const uint32_t v = V[i], S = 32u + (in ? ti : 0u);
          const bool low = v + S < c;
          lows |= low;
          amb |= !low && v < c + sum;
          if (in) {
            sv()[gi] = low ? make_uint2(v, S) : make_uint2(0u, (uint32_t)i);
            Ig |= 1u << gi;
            if (low) Lg |= 1u << gi;
          }
        }
      }
      __syncwarp();
      if (!__any_sync(KCL_FULL, amb)) {
        if (!__any_sync(KCL_FULL, lows)) {
          c += sum;
          continue;
        }
        Lg = __reduce_or_sync(KCL_FULL, Lg);
        uint32_t ng_taken = 0, taken = 0;  // lane g: takers of u_g's chain, u_g in L
        bool clash = false;
        for (int q = 0; q < ns; ++q) {
          const int i = 32 * q + lane;
          const int j = i < ni ? (int)il[i] : a + 64;
          const bool in = j >= a && j < a + ng;
          const uint32_t ti = __shfl_sync(KCL_FULL, tot, j & 31);
          const uint32_t v = i < ni ? V[i] : 0x7fffffffu, S = 32u + (in ? ti : 0u);
          const bool low = j < a + ng && v + S < c;
          uint32_t inc = 0;
          if (__any_sync(KCL_FULL, low)) {
            uint32_t T = column_bits(rows, ro(), i < ni ? list()[j] : 0u, j, a, ng);
            if (!low) T = 0;  // the others always fall
            inc = (uint32_t)__popc(T & ~Lg);
            taken += inc;
            for (uint32_t rem = Lg; rem; rem &= rem - 1) {
              const int g = __ffs(rem) - 1;
              const uint2 x = sv()[g];
              const bool has = (T >> g) & 1u, take = has && v + S < x.x;
              clash |= has && !take && v < x.x + x.y;
              const uint32_t n = (uint32_t)__popc(__ballot_sync(KCL_FULL, take));
              if (lane == g) ng_taken += n;
              inc += take;
            }
          }
          if (i < ni) I8[i] = (uint8_t)inc;
        }
        if (!__any_sync(KCL_FULL, clash)) {
          const uint32_t fell = ((Lg >> lane) & 1u) ? tot - ng_taken : 0u;
          for (int q = 0; q < ns; ++q) {
            const int i = 32 * q + lane;
            const int gi = i < ni ? (int)il[i] - a : 64;
            const uint32_t f = __shfl_sync(KCL_FULL, fell, gi & 31);
            if (i < ni) V[i] += I8[i] + (gi >= 0 && gi < ng ? f : 0u);
          }
          c += __reduce_add_sync(KCL_FULL, (((Lg >> lane) & 1u) ? 0u : tot) - taken);
          continue;
        }
        // the chains need the members' places, not their values
        __syncwarp();
        for (int q = 0; q < ns; ++q) {
          const int i = 32 * q + lane;
          const int gi = i < ni ? (int)il[i] - a : 64;
          if (gi >= 0 && gi < ng) sv()[gi].y = (uint32_t)i;
        }
        __syncwarp();
      } else if (__any_sync(KCL_FULL, Lg != 0)) {
        for (int q = 0; q < ns; ++q) {
          const int i = 32 * q + lane;
          const int gi = i < ni ? (int)il[i] - a : 64;
          if (gi >= 0 && gi < ng) sv()[gi].y = (uint32_t)i;
        }
        __syncwarp();
      }
      Ig = __reduce_or_sync(KCL_FULL, Ig);
      for (uint32_t rem = __ballot_sync(KCL_FULL, tot != 0); rem; rem &= rem - 1) {
        const int g = __ffs(rem) - 1;
        const uint32_t og = ro()[g];
        const uint32_t tu = __shfl_sync(KCL_FULL, tot, g);
        uint32_t vu = 0x7fffffffu, iu = 0;
        if ((Ig >> g) & 1u) {
          iu = sv()[g].y;
          __syncwarp();  // the value is its own lane's
          vu = V[iu];
        }
        const bool own = vu < c;  // strict: ties stay with the earlier argmin
        const uint32_t c0 = own ? vu : c;
        uint32_t n = 0;  // takers
        if (dense) {
          uint32_t cl = c0;
          for (int i0 = 0; i0 < a + g; i0 += 32) {
            const int i = i0 + lane;
            bool has = false;
            uint32_t v = 0;
            if (i < a + g) {
              const uint32_t id = list()[i];
              has = (rows[og + (id >> 5)] >> (id & 31)) & 1u;
              v = V[i];
            }
            if ((takers_dense(has, v, cl, lt) >> lane) & 1u) V[i] = v + 1u;
          }
          n = tu - (cl - c0);
        } else {
          bool near = false;
          uint32_t hasq = 0;
          for (int q = 0; q < ns; ++q) {
            const int i = 32 * q + lane;
            const int j = i < ni ? (int)il[i] : a + 64;
            if (j < a + g) {
              const uint32_t id = list()[j];
              if ((rows[og + (id >> 5)] >> (id & 31)) & 1u) {
                hasq |= 1u << q;
                near |= V[i] - c0 < tu;
              }
            }
          }
          if (!__any_sync(KCL_FULL, near)) {
            for (int q = 0; q < ns; ++q)
              if ((hasq >> q) & 1u) {
                const int i = 32 * q + lane;
                const uint32_t v = V[i], t = (v - c0) >> 31;
                V[i] = v + t;
                n += t;
              }
            n = __reduce_add_sync(KCL_FULL, n);
          } else {
            uint32_t Q, pre;
            words_of(list()[a + g], og, Q, pre);
            for (int q = 0; q < ns; ++q) {
              const int i = 32 * q + lane;
              const bool has = (hasq >> q) & 1u;
              const uint32_t id = has ? list()[il[i]] : 0u;
              const uint32_t v = has ? V[i] : 0u;
              const uint32_t mk = takers_sparse(has, v, c0, ahead_of(id, Q, pre), n, lt);
              if ((mk >> lane) & 1u) V[i] = v + 1u;
              n += (uint32_t)__popc(mk);
            }
          }
        }
        const uint32_t fell = tu - n;
        if (!own) c += fell;
        else if (lane == (int)(iu & 31u)) V[iu] += fell;
      }
    }
    for (int i = lane; i < ni; i += 32) {
      const uint32_t id = list()[il[i]];
      put(id, ACC ? val[id] : 0u, V[i]);
    }
    __syncwarp();
    return c;
  }

  // The two levels over P (lane w: word w) from prefix value c.  Returns
  // false, with nothing changed, when I outgrows the scratch.
  __device__ __forceinline__ bool operator()(uint32_t P, uint32_t &c) const {
    const uint32_t lt = lanemask_lt();
    __syncwarp();
    pw()[lane] = P;
    const int np = list_members(P, list(), lane);
    if (np < 2) return true;
    __syncwarp();
    if (np <= 32) {  // one slot holds P: choosing I would cost more than it saves
      c = run1<true>(np, np, c);
      return true;
    }
    const uint32_t reach = c + (uint32_t)np * (uint32_t)(np - 1) / 2u;
    int ni = 0;
    for (int b = 0; b < np; b += 32) {
      const bool in = b + lane < np && val[list()[b + lane]] < reach;
      const uint32_t mk = __ballot_sync(KCL_FULL, in);
      const int p = ni + __popc(mk & lt);
      if (in && p < kPairMembers) ilist()[p] = (uint16_t)(b + lane);
      ni += __popc(mk);
    }
    if (ni <= 32) {
      __syncwarp();
      c = run1<false>(np, ni, c);
      return true;
    }
    if (2 * ni > np && np <= kPairMembers) {  // then I = P: no members between
      for (int i = lane; i < np; i += 32) ilist()[i] = (uint16_t)i;
      ni = np;
    }
    if (ni > kPairMembers) return false;
    __syncwarp();
    c = run_slots(np, ni, c);
    return true;
  }
};

// Level L of a root-edge stream over candidates P with prefix argmin g of
// current value cg (kCDensestNoAtom.c:173-188 for L = 2, 237-259 above).
// Returns g's new value; the argmin of a deeper prefix, when it is u, is
// written back by u's lane.  SKIP (one word per lane, 32-bit values): the
// last level runs chain_word1 with lo, the per-word lower bounds.  PAIR (the
// same, private values): the last two levels run as one PairLevel, and one
// word at a time only when that has no room (pair: its scratch).
template <int L, int WPL, typename VA, bool SKIP, bool PAIR = false>
__device__ __forceinline__ typename VA::T seq_rec(const Bits<WPL> &P, typename VA::T cg, const uint32_t *rows,
                                                  const VA &va, typename VA::T lo, int lane, uint32_t *err,
                                                  uint32_t *pair = nullptr) {
  using T = typename VA::T;
  if constexpr (PAIR && L == 2) {
    static_assert(WPL == 1 && SKIP, "the pair level needs one word per lane and 32-bit values");
    if (PairLevel<false>{rows, va.cur, nullptr, pair, lane}(P.w[0], cg)) return cg;
    lo = 0xffffffffu;
    uint32_t nz = __ballot_sync(KCL_FULL, P.w[0] != 0);
    while (nz) {
      const int w = __ffs(nz) - 1;
      nz &= nz - 1;
      const uint32_t word = __shfl_sync(KCL_FULL, P.w[0], w);
      const uint32_t val = __reduce_min_sync(KCL_FULL, ((word >> lane) & 1u) ? va.cur[(w << 5) | lane] : 0xffffffffu);
      if (lane == w) lo = val;
    }
    return seq_rec<2, 1, VA, true, false>(P, cg, rows, va, lo, lane, err);
  } else if constexpr (L == 1) {
    if constexpr (SKIP) {
      static_assert(WPL == 1 && sizeof(T) == 4, "the word skip needs one word per lane and 32-bit values");
      return chain_word1<VA>(P.w[0], cg, va, lo, lane, err);
    } else {
      return chain_words<WPL, VA>(P, cg, va, lane, err);
    }
  } else if constexpr (WPL == 1) {
    if constexpr (L >= 3) {
      const uint32_t pc = __reduce_add_sync(KCL_FULL, (uint32_t)__popc(P.w[0]));  // kCDensestNoAtom.c:218
      if (pc < (uint32_t)L) return cg;
    }
    // The members u of P in ascending order, word a of P at a time.  Row u =
    // 32 a + b keeps a + 1 words, packed from tri_off(32 a) = 16 a (a + 1)
    // with a stride of a + 1 words between the rows of word a.
    uint32_t nzw = __ballot_sync(KCL_FULL, P.w[0] != 0);
    while (nzw) {
      const int a = __ffs(nzw) - 1;
      nzw &= nzw - 1;
      uint32_t wb = __shfl_sync(KCL_FULL, P.w[0], a);
      const uint32_t stride = (uint32_t)a + 1u;
      const uint32_t *row0 = rows + 16u * (uint32_t)a * stride + (uint32_t)lane;
      const bool in_row = lane <= a;
      while (wb) {
        const int b = __ffs(wb) - 1;
        wb &= wb - 1;
        const int u = (a << 5) | b;
        // u's value: its word is written by lane b only; the warp barrier
        // orders those writes before every lane's read.
        __syncwarp();
        uint32_t raw;
        const T vu = va.get(u, raw);
        const bool take = vu < cg;  // strict: ties stay with the earlier argmin
        Bits<1> Q;
        Q.w[0] = in_row ? (P.w[0] & row0[(uint32_t)b * stride]) : 0u;
        const T c0 = take ? vu : cg;
        const T c1 = seq_rec<L - 1, 1, VA, SKIP, PAIR>(Q, c0, rows, va, lo, lane, err, pair);
        if (take) {
          if (lane == b) va.add(u, c1 - c0, err);
        } else {
          cg = c1;
        }
      }
    }
    return cg;
  } else {
    if constexpr (L >= 3) {
      const int pc = warp_sum(popc_lane(P));  // kCDensestNoAtom.c:218
      if (pc < L) return cg;
    }
    for_each_bit<WPL>(P, [&](int u) {
      const T vu = value_of<VA>(u, va, lane);
      const bool take = vu < cg;  // strict: ties stay with the earlier argmin
      const Bits<WPL> Q = band(P, load_row<WPL, true>(rows, u, 0, lane));
      const T c0 = take ? vu : cg;
      const T c1 = seq_rec<L - 1, WPL, VA, SKIP>(Q, c0, rows, va, lo, lane, err);
      if (take) {
        if (lane == (u & 31)) va.add(u, c1 - c0, err);
      } else {
        cg = c1;
      }
    });
    return cg;
  }
}

// Apply f(i) on the lane owning each member i of C (lane i & 31).
template <int WPL, typename F>
__device__ __forceinline__ void for_members(const Bits<WPL> &C, int lane, F &&f) {
#pragma unroll
  for (int qq = 0; qq < WPL; ++qq) {
    uint32_t nz = __ballot_sync(KCL_FULL, C.w[qq] != 0);
    while (nz) {
      const int L = __ffs(nz) - 1;
      nz &= nz - 1;
      const uint32_t word = __shfl_sync(KCL_FULL, C.w[qq], L);
      if ((word >> lane) & 1u) f(((L + 32 * qq) << 5) | lane);
    }
  }
}

// A stream over the nc candidates C on the root's 32-bit values.  False, with
// nothing done, when a prefix value it can reach comes near their cap (see
// kRelCap), or its followed members outgrow the scratch.
template <int K>
__device__ __forceinline__ bool stream_on_rel(const Bits<1> &C, uint32_t nc, int g0, const uint32_t *rows,
                                              const uint32_t *rel, uint32_t *cur, unsigned long long *acc,
                                              uint32_t *pair, int lane, uint32_t *err) {
  unsigned long long bound = 1;  // C(nc, K - 2): the stream's cliques at most
#pragma unroll
  for (uint32_t i = 0; i < (uint32_t)(K - 2); ++i) bound = bound * (nc - i) / (i + 1u);
  const uint32_t c0 = rel[g0];
  if (bound + 64 >= (unsigned long long)(kRelCap - c0)) return false;
  uint32_t c = c0;
  if constexpr (K == 3) {
    // One chain: nothing reads a value twice, so the takers' units go straight
    // to acc.
    const uint32_t lt = lanemask_lt();
    uint32_t nz = __ballot_sync(KCL_FULL, C.w[0] != 0);
    while (nz) {
      const int w = __ffs(nz) - 1;
      nz &= nz - 1;
      const uint32_t word = __shfl_sync(KCL_FULL, C.w[0], w);
      const bool has = (word >> lane) & 1u;
      const int v = (w << 5) | lane;
      const uint32_t m = word_fixed_point(has ? (int)(rel[v] - c) : -1, lt);
      if (has && !((m >> lane) & 1u)) shared_add(acc + v, 1u);
      c += (uint32_t)__popc(m);
    }
  } else if (nc <= (K == 4 ? 32u : 64u)) {
    // Two slots cost 64 column reads per member up front: k = 4, with one pair
    // of levels per stream, has nothing to spread them over.
    uint16_t *list = PairLevel<true>{nullptr, nullptr, nullptr, pair, lane}.list();
    __syncwarp();
    list_members(C.w[0], list, lane);
    __syncwarp();
    if (K == 4 || nc <= 32) {
      TinyStream<1> ts;
      ts.lane = lane;
      c = ts.template run<K>(rows, list, (int)nc, rel, acc, c);
    } else {
      TinyStream<2> ts;
      ts.lane = lane;
      c = ts.template run<K>(rows, list, (int)nc, rel, acc, c);
    }
  } else if constexpr (K == 4) {
    if (!PairLevel<true>{rows, const_cast<uint32_t *>(rel), acc, pair, lane}(C.w[0], c)) return false;
  } else {
    for_members<1>(C, lane, [&](int i) { cur[i] = rel[i]; });
    const Vals32 va{cur};
    c = seq_rec<K - 2, 1, Vals32, true, true>(C, c, rows, va, 0u, lane, err, pair);
    __syncwarp();
    for_members<1>(C, lane, [&](int i) {
      const uint32_t delta = cur[i] - rel[i];
      if (delta) shared_add(&acc[i], delta);
    });
  }
  if (lane == 0 && c != c0) shared_add(&acc[g0], c - c0);
  return true;
}

// A root's sub-task counter: sub-tasks taken below, CTAs that joined it above.
constexpr int kTaskBits = 20;  // 2048 sub-tasks and one overshoot per warp of 2048 CTAs
constexpr uint32_t kTaskMask = (1u << kTaskBits) - 1u;

// A stream on 64-bit values at k >= 6 (its values differ by 2^31 or more).  A
// function of its own, so that its recursion does not share its registers with
// what the other streams keep: loads spread over 2^40, us a pass inlined and so,
// planted RMAT-12 at k = 6 2906 and 2482, Chung-Lu 3,000 at k = 8 4441 and 3295;
// no difference for loads within 2^31.
template <int K>
__device__ __noinline__ void stream_wide(uint32_t word, int g0, const uint32_t *rows, const unsigned long long *base,
                                         uint32_t *cur, unsigned long long *acc, int lane, uint32_t *err) {
  Bits<1> C;
  C.w[0] = word;
  for_members<1>(C, lane, [&](int i) { cur[i] = 0; });
  const Vals64<true> va{base, cur};
  const unsigned long long c0 = base[g0];
  const unsigned long long c1 = seq_rec<K - 2, 1, Vals64<true>, false>(C, c0, rows, va, 0u, lane, err);
  for_members<1>(C, lane, [&](int i) {
    const uint32_t delta = cur[i];
    if (delta) shared_add(&acc[i], delta);
  });
  if (lane == 0 && c1 != c0) shared_add(&acc[g0], c1 - c0);
}

// Every root-edge stream of the current root, the warp taking streams from
// the root's shared counter (largest candidate sets first); increments go to
// the CTA's acc[] (kCDensestNoAtom.c:270-295 per root edge).
//
// Rows in shared memory: the streams read rel, the root's values as
// 32-bit offsets from the smallest of them capped at kRelCap; a stream whose
// prefix value cannot reach the cap uses them (a capped member then lies above
// every prefix value, so the cap changes no comparison).  Otherwise the
// stream makes its own values:
//
// A stream's values fit the 32-bit form when, with off = the smallest
// pass-start value among {s, t} and C and cap = (the edge argmin's value
// - off) + the most increments one vertex can take in the stream + 64, cap
// stays below 2^31: values above cap are stored as cap, which changes no
// comparison -- the prefix value never exceeds cap - 64, so such a candidate
// falls to the prefix whatever came before it (its distance is >= 64 > 31),
// and it never becomes the prefix argmin.
template <int K, int WPL>
__device__ __forceinline__ void seq_streams(uint32_t *next, int d, const uint32_t *rows,
                                            const unsigned long long *base, uint32_t *cur,
                                            unsigned long long *acc, const uint32_t *rel, uint32_t *pair, int lane,
                                            uint32_t *err) {
  for (;;) {
    int q = 0;
    if (lane == 0) q = (int)(atomicAdd(next, 1u) & kTaskMask);
    q = __shfl_sync(KCL_FULL, q, 0);
    if (q >= d) break;
    const int j = d - 1 - q;
    const Bits<WPL> C = load_row<WPL, true>(rows, j, 0, lane);
    if (!any_bits<WPL>(C)) continue;
    const int g0 = base[j] < base[d] ? j : d;  // kCDensestNoAtom.c:287
    if constexpr (WPL == 1) {
      const uint32_t nc = __reduce_add_sync(KCL_FULL, (uint32_t)__popc(C.w[0]));
      if (nc < (uint32_t)(K - 2)) continue;
      if (stream_on_rel<K>(C, nc, g0, rows, rel, cur, acc, pair, lane, err)) continue;
      if constexpr (K >= 6) {
        stream_wide<K>(C.w[0], g0, rows, base, cur, acc, lane, err);
        continue;
      }
    }
    bool r32 = false;
    unsigned long long off = 0, cap = 0;
    if constexpr (K <= 5) {
      unsigned long long lo = base[g0];
      int nc = 0;
      for_members<WPL>(C, lane, [&](int i) {
        const unsigned long long b = base[i];
        lo = b < lo ? b : lo;
        ++nc;
      });
      lo = warp_min_u64(lo);
      nc = warp_sum(nc);
      unsigned long long bound = 1;  // C(nc, K - 2) >= the increments of one vertex
      for (int i = 0; i < K - 2; ++i) bound = bound * (unsigned long long)(nc - i) / (unsigned long long)(i + 1);
      off = lo;
      cap = (base[g0] - lo) + bound + 64;
      r32 = cap < 0x7fffffffull;
    }
    if (r32) {
      // Stored values, and per word of C the smallest of them (lane = word).
      uint32_t lo = 0xffffffffu;
#pragma unroll
      for (int qq = 0; qq < WPL; ++qq) {
        uint32_t nz = __ballot_sync(KCL_FULL, C.w[qq] != 0);
        while (nz) {
          const int L = __ffs(nz) - 1;
          nz &= nz - 1;
          const uint32_t word = __shfl_sync(KCL_FULL, C.w[qq], L);
          uint32_t val = 0xffffffffu;
          if ((word >> lane) & 1u) {
            const int i = ((L + 32 * qq) << 5) | lane;
            const unsigned long long rel = base[i] - off;
            val = (uint32_t)(rel < cap ? rel : cap);
            cur[i] = val;
          }
          val = __reduce_min_sync(KCL_FULL, val);
          if (qq == 0 && lane == L) lo = val;
        }
      }
      const Vals32 va{cur};
      const uint32_t c0 = (uint32_t)(base[g0] - off);
      const uint32_t c1 = seq_rec<K - 2, WPL, Vals32, (WPL == 1)>(C, c0, rows, va, lo, lane, err);
      for_members<WPL>(C, lane, [&](int i) {
        const unsigned long long rel = base[i] - off;
        const uint32_t delta = cur[i] - (uint32_t)(rel < cap ? rel : cap);
        if (delta) shared_add(&acc[i], delta);
      });
      if (lane == 0 && c1 != c0) shared_add(&acc[g0], c1 - c0);
    } else {
      for_members<WPL>(C, lane, [&](int i) { cur[i] = 0; });
      const Vals64<(K >= 6)> va{base, cur};
      const unsigned long long c0 = base[g0];
      const unsigned long long c1 = seq_rec<K - 2, WPL, Vals64<(K >= 6)>, false>(C, c0, rows, va, 0u, lane, err);
      for_members<WPL>(C, lane, [&](int i) {
        const uint32_t delta = cur[i];
        if (delta) shared_add(&acc[i], delta);
      });
      if (lane == 0 && c1 != c0) shared_add(&acc[g0], c1 - c0);
    }
  }
}

// KCLPP_SEQ_SHARED: every root-edge stream of the current root against the
// pass's one load vector r (updated in place).  When a stream starts, the
// CTA's copy of its vertices' values is raised to r's (relative to off, the
// root's smallest value when it started); the chain is the reference's
// (kCDensestNoAtom.c:155-268) on the copy plus the stream's own increments;
// when it closes, its increments go to the copy (seen at once by the CTA's
// other streams) and, by atomic adds, to r (seen by every stream that starts
// later).  Every clique still gives exactly one unit to one of its members,
// so r / T stays a feasible load whatever the interleaving; which member
// gets it depends on the timing of the other streams (not deterministic).
// The vector is read and added to once per stream and vertex, not per
// clique: the whole GPU reading a few kilobytes of L2 at every candidate
// serialises on the few L2 slices that hold them.
template <int K, int WPL>
__device__ __forceinline__ void seq_streams_shared(uint32_t *next, int d, const uint32_t *rows, const uint32_t *list,
                                                   uint32_t s, unsigned long long *r, unsigned long long off,
                                                   uint32_t *cur, uint32_t *dl, int lane, uint32_t *err) {
  const ValsShared va{cur, dl};
  auto id = [&](int i) { return i < d ? list[i] : s; };
  auto refresh = [&](int i) {
    const unsigned long long v = __ldcg(r + id(i)) - off;
    atomicMax(cur + i, v < kSharedCap ? (uint32_t)v : kSharedCap);
  };
  auto close = [&](int i, uint32_t x) {
    atomicAdd(cur + i, x);
    atomicAdd(r + id(i), (unsigned long long)x);
  };
  for (;;) {
    int q = 0;
    if (lane == 0) q = (int)(atomicAdd(next, 1u) & kTaskMask);
    q = __shfl_sync(KCL_FULL, q, 0);
    if (q >= d) break;
    const int j = d - 1 - q;
    const Bits<WPL> C = load_row<WPL, true>(rows, j, 0, lane);
    if (!any_bits<WPL>(C)) continue;
    // Refresh the members' values and take, per word of C (lane = word), the
    // smallest of them: values only grow while the stream runs, so a word
    // whose candidates all start at or above the prefix's reach falls to the
    // prefix whole (the chain's skip).
    uint32_t lo = 0xffffffffu;
#pragma unroll
    for (int qq = 0; qq < WPL; ++qq) {
      uint32_t nz = __ballot_sync(KCL_FULL, C.w[qq] != 0);
      while (nz) {
        const int L = __ffs(nz) - 1;
        nz &= nz - 1;
        const uint32_t word = __shfl_sync(KCL_FULL, C.w[qq], L);
        uint32_t val = 0xffffffffu;
        if ((word >> lane) & 1u) {
          const int i = ((L + 32 * qq) << 5) | lane;
          refresh(i);
          dl[i] = 0;
          val = *(volatile uint32_t *)(cur + i);
        }
        val = __reduce_min_sync(KCL_FULL, val);
        if (qq == 0 && lane == L) lo = val;
      }
    }
    uint32_t vj = 0, vd = 0;
    if (lane == 0) {
      refresh(j);
      refresh(d);
      vj = *(volatile uint32_t *)(cur + j);
      vd = *(volatile uint32_t *)(cur + d);
    }
    __syncwarp();
    const int g0 = __shfl_sync(KCL_FULL, vj < vd ? j : d, 0);  // kCDensestNoAtom.c:287
    const uint32_t c0 = __shfl_sync(KCL_FULL, vj < vd ? vj : vd, 0);
    const uint32_t c1 = seq_rec<K - 2, WPL, ValsShared, (WPL == 1)>(C, c0, rows, va, lo, lane, err);
    for_members<WPL>(C, lane, [&](int i) {
      const uint32_t x = dl[i];
      if (x) close(i, x);
    });
    if (lane == 0 && c1 != c0) close(g0, c1 - c0);
  }
}

// A root's induced rows (MakeSubgraph's induced adjacency,
// kCDensestNoAtom.c:104-113), one warp per row i: the members of list[0, i)
// that are out-neighbours of list[i].  A member with a bitmap row is asked
// about 32 earlier members at a time: word(i, w, hit), all lanes, the lane's
// member being 32 w + lane; the others' out-lists are walked, a lane per
// out-neighbour, and looked up in the table: pair(i, j) on the finding lane.
// Latency bounds this phase (a row's offsets, its list and the look-ups are
// dependent reads), and it was 42 to 68 % of a CTA's time once the streams were
// cheap: walking every list with a binary search, the k = 3 wave passes of an
// RMAT-17 graph took 6.0 ms, now 3.2; the k = 4 count of RMAT-18 4.1 -> 2.2 ms,
// a Seq pass over the RMAT-18 core 1.36 -> 1.03 ms.
template <typename Word, typename Pair>
__device__ __forceinline__ void induce_rows(const PassArgs &a, const uint32_t *list, int d, const uint32_t *tab, int tb,
                                            int wid, int nwarps, int lane, Word &&word, Pair &&pair) {
  for (int r0 = wid; r0 < d; r0 += nwarps * 32) {
    // this warp's next 32 rows: r0, r0 + nwarps, ...
    const int ri = r0 + nwarps * lane;
    const uint4 br = ri < d ? bit_row(a, list[ri]) : make_uint4(kNoBitRow, 0u, 0u, 0u);
    for (int q = 0, i = r0; q < 32 && i < d; ++q, i += nwarps) {
      const uint32_t bo = __shfl_sync(KCL_FULL, br.x, q), bf = __shfl_sync(KCL_FULL, br.y, q);
      const uint32_t bs = __shfl_sync(KCL_FULL, br.z, q);
      if (i == 0) continue;
      if (bo != kNoBitRow) {
        const int nw = (i + 31) >> 5;
#pragma unroll 4
        for (int w = 0; w < nw; ++w) {
          const int j = (w << 5) | lane;
          word(i, w, j < i && bit_at(a, bo, bf, bs, list[j]));
        }
        continue;
      }
      const uint32_t x = list[i];
      const uint32_t top = list[i - 1];
      const uint64_t xe = a.off[x + 1];
      for (uint64_t e = a.off[x] + lane; e < xe; e += 32) {
        const uint32_t y = a.cols[e];
        if (y > top) break;  // ascending: no later neighbour is in list[0, i)
        const int j = tab_find(tab, tb, list, y);
        if (j >= 0) pair(i, j);
      }
      __syncwarp();
    }
  }
}

// Work stealing: once the root list is exhausted, an idle CTA joins a root
// whose sub-tasks (root edges or rows) are not all taken, rebuilds that root's
// G_s and takes sub-tasks from the same global counter.  Every CTA publishes
// the root it holds (plus one; 0: none) in its slot of a.active; the thief's
// threads look at a slot each and the CTA joins the root with the most
// sub-tasks left per CTA on it, if that is at least steal_quarters of its warps
// -- below, rebuilding the rows costs more than the share saves.  A root's
// counter holds the sub-tasks taken in its low kTaskBits and the CTAs that
// joined above.  (One warp scanning, every CTA joining the root with most left:
// a Seq pass over the RMAT-18 core took 858 us, now 482.)
// Least share in quarters of the CTA's warps: a sub-task grows with k.
template <int MODE, int K>
constexpr uint32_t steal_quarters() { return MODE == MODE_SEQ && K >= 5 ? 1 : 4; }
template <bool IDENT>
__device__ __forceinline__ uint32_t find_victim(const PassArgs &a, int need, uint32_t least, uint32_t *s_best,
                                                uint32_t *s_who) {
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5, nw = (int)(blockDim.x >> 5);
  uint32_t best = 0, best_idx = UINT32_MAX;
  for (uint32_t b = tid; b < gridDim.x; b += blockDim.x) {
    const uint32_t held = __ldcg(a.active + b);
    if (held == 0 || held > a.num_roots) continue;
    const uint32_t idx = held - 1;
    const uint32_t s = IDENT ? idx : a.roots[idx];
    const uint32_t d = a.list_off ? (uint32_t)(a.list_off[s + 1] - a.list_off[s]) : (uint32_t)(a.off[s + 1] - a.off[s]);
    const uint32_t t = __ldcg(a.task_next + idx), taken = t & kTaskMask;
    const bool in_window = !IDENT || (d >= a.deg_lo && d <= a.deg_hi && d <= a.dmax);
    if (!in_window || (int)d < need || d < a.steal_min || taken >= d) continue;
    const uint32_t share = (d - taken) / ((t >> kTaskBits) + 2u);  // with its owner, those who joined, and this CTA
    if (share >= least && share > best) {
      best = share;
      best_idx = idx;
    }
  }
  const uint32_t top = __reduce_max_sync(KCL_FULL, best);
  const uint32_t who = __ballot_sync(KCL_FULL, best == top);
  const uint32_t idx = __shfl_sync(KCL_FULL, best_idx, __ffs(who) - 1);
  if (lane == 0) {
    s_best[wid] = top;
    s_who[wid] = idx;
  }
  __syncthreads();
  const uint32_t mine = lane < nw ? s_best[lane] : 0u;
  const uint32_t all = __reduce_max_sync(KCL_FULL, mine);
  if (all == 0) return UINT32_MAX;
  return s_who[__ffs(__ballot_sync(KCL_FULL, mine == all)) - 1];
}

// Register budget of a tier M / L kernel, as CTAs of the widest launch
// (warps_m) that must fit one SM: two for the Seq kernels, whose widest launch
// narrows as k grows (40 registers a thread at k <= 4, 64 at k = 5, 6, 80
// beyond), and for the shallow counting kernels (<= 32 at k <= 4, <= 42 at
// k = 5 with 24-warp CTAs); one for the deeper counting kernels, which would
// otherwise spill.
template <int MODE, int K>
constexpr int min_ctas_m() { return MODE == MODE_SEQ || K <= 5 ? 2 : 1; }

template <int MODE, int K, int WPL, bool ROWS_IN_SMEM, bool IDENT = false>
__global__ void __launch_bounds__(warps_m<MODE, K>() * 32, min_ctas_m<MODE, K>()) tier_m_kernel(PassArgs a) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int NW = (int)(blockDim.x >> 5);
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  const int dmax = (int)a.dmax;
  const LayoutM lay = layout_m(MODE, K, a.dmax, NW, ROWS_IN_SMEM);
  uint32_t *list = reinterpret_cast<uint32_t *>(smem_raw + lay.list);
  uint32_t *tab = reinterpret_cast<uint32_t *>(smem_raw + lay.tab);
  uint32_t *rows = ROWS_IN_SMEM ? reinterpret_cast<uint32_t *>(smem_raw + lay.rows)
                                : a.slab + (size_t)blockIdx.x * a.slab_words;
  unsigned long long *base = reinterpret_cast<unsigned long long *>(smem_raw + lay.base);
  unsigned long long *acc = reinterpret_cast<unsigned long long *>(smem_raw + lay.acc);
  uint16_t *rank = reinterpret_cast<uint16_t *>(smem_raw + lay.rank);
  uint16_t *inv = reinterpret_cast<uint16_t *>(smem_raw + lay.inv);
  uint32_t *dl = reinterpret_cast<uint32_t *>(smem_raw + lay.dl) + (size_t)wid * seq_warp_words(K, a.dmax, ROWS_IN_SMEM);
  uint32_t *pair = K == 4 ? dl : dl + ((size_t)dmax + 4) / 4 * 4;
  uint32_t *rel = reinterpret_cast<uint32_t *>(smem_raw + lay.rel);
  uint32_t *cbuf = reinterpret_cast<uint32_t *>(smem_raw + lay.cbuf) + (size_t)wid * cbuf_words(K, a.dmax);

  __shared__ uint32_t s_idx, s_best[32], s_who[32];
  __shared__ int s_tau;
  __shared__ unsigned long long s_sum;
  __shared__ unsigned long long s_off;  // Seq: the root's smallest value

  if constexpr (MODE == MODE_SEQ) {
    for (int i = tid; i <= dmax; i += NW * 32) acc[i] = 0;
    for (int i = lane; i <= dmax; i += 32) dl[i] = 0;
  }
  __shared__ unsigned long long s_min[MODE == MODE_SEQ ? 32 : 1];
  // The CTA's smallest x (a warp's share each; one barrier).
  auto cta_min = [&](unsigned long long x) {
    x = warp_min_u64(x);
    if (lane == 0) s_min[wid] = x;
    __syncthreads();
    return warp_min_u64(lane < NW ? s_min[lane] : ~0ull);
  };
  bool stealing = false;
  __syncthreads();
  for (;;) {
    uint32_t idx;
    if (tid == 0) {
      if (!stealing) s_idx = atomicAdd(a.work, 1u);
      s_tau = 0;
      s_sum = 0;
    }
    if (!stealing) {
      __syncthreads();
      idx = s_idx;
      stealing = idx >= a.num_roots;
    }
    if (stealing) {
      if (!a.active) break;
      const uint32_t least = a.shared_loads ? 2u : ((uint32_t)NW * steal_quarters<MODE, K>() + 3u) / 4u;
      idx = find_victim<IDENT>(a, K - 1, least > 2u ? least : 2u, s_best, s_who);
      if (idx == UINT32_MAX) break;
      if (tid == 0) atomicAdd(a.task_next + idx, 1u << kTaskBits);
    }
    if (tid == 0 && a.active) a.active[blockIdx.x] = idx + 1;  // visible to thieves
    uint32_t *next = a.task_next + idx;  // root's sub-task counter, shared by every CTA on it
    const uint32_t s = IDENT ? idx : a.roots[idx];
    uint64_t o;
    int d;
    const uint32_t *lcols;
    if constexpr (MODE == MODE_COUNT) {
      root_span(a, s, o, d, lcols);
    } else {
      o = a.off[s];
      d = (int)(a.off[s + 1] - o);
      lcols = a.cols;
    }
    if constexpr (IDENT) {
      if ((uint32_t)d < a.deg_lo || (uint32_t)d > a.deg_hi) {
        __syncthreads();
        continue;
      }
    }
    if (d > dmax || d > 32 * 32 * WPL) {
      if (tid == 0) { atomicOr(a.err, ERR_DEGREE); atomicMax(next, (uint32_t)d); }
      __syncthreads();
      continue;
    }
    if (d < K - 1 || d == 0) {
      __syncthreads();
      continue;
    }
    const int W = (d + 31) >> 5;
    const int row_words = MODE == MODE_SEQ ? (int)tri_off((uint32_t)d) : d * W;
    for (int i = tid; i < d; i += NW * 32) list[i] = lcols[o + i];
    for (int i = tid; i < row_words; i += NW * 32) rows[i] = 0;
    const int tb = tab_bits((uint32_t)d);
    for (int i = tid; i < 1 << tb; i += NW * 32) tab[i] = kTabEmpty;
    if constexpr (MODE == MODE_ORDER) {
      for (int i = tid; i < d; i += NW * 32) base[i] = vertex_key(a, a.cols[o + i]);
      if (tid == 0) base[d] = vertex_key(a, s);
    }
    if constexpr (MODE == MODE_SEQ) {
      if (a.shared_loads) {
        // The load vector as it is now (from L2: other SMs add to it), as 32-bit
        // values relative to its smallest entry among the root's vertices, in
        // the acc array (which this mode does not otherwise use).
        uint32_t *cur = reinterpret_cast<uint32_t *>(acc);
        unsigned long long mn = ~0ull;
        for (int i = tid; i <= d; i += NW * 32) {
          base[i] = __ldcg(a.out + (i < d ? a.cols[o + i] : s));
          mn = base[i] < mn ? base[i] : mn;
        }
        const unsigned long long off = cta_min(mn);
        if (tid == 0) s_off = off;
        for (int i = tid; i <= d; i += NW * 32) {
          const unsigned long long v = base[i] - off;
          cur[i] = v < kSharedCap ? (uint32_t)v : kSharedCap;
        }
      } else {
        unsigned long long mn = ~0ull;
        for (int i = tid; i <= d; i += NW * 32) {
          const unsigned long long v = a.r_in[i < d ? a.cols[o + i] : s];
          base[i] = v;
          mn = v < mn ? v : mn;
        }
        if constexpr (ROWS_IN_SMEM) {
          const unsigned long long off = cta_min(mn);
          for (int i = tid; i <= d; i += NW * 32) {
            const unsigned long long v = base[i] - off;
            rel[i] = v < kRelCap ? (uint32_t)v : kRelCap;
          }
        }
      }
    }
    __syncthreads();
    if constexpr (MODE == MODE_ORDER) {
      const unsigned long long ks = base[d];
      int t = 0;
      for (int i0 = wid * 32; i0 < d; i0 += NW * 32) {
        // keys at or below i's before it, below i's after it: one comparison
        // each but among the warp's own 32
        const int i = i0 + lane;
        const unsigned long long ki = i < d ? base[i] : 0ull;
        const int mid = i0 + 32 < d ? i0 + 32 : d;
        int r = 0;
#pragma unroll 4
        for (int j = 0; j < i0; ++j) r += base[j] <= ki;
        for (int j = i0; j < mid; ++j) {
          const unsigned long long kj = base[j];
          r += (kj < ki) || (kj == ki && j < i);
        }
#pragma unroll 4
        for (int j = mid; j < d; ++j) r += base[j] < ki;
        if (i >= d) continue;
        rank[i] = (uint16_t)r;
        inv[r] = (uint16_t)i;
        t += (ki <= ks);
      }
      t = warp_sum(t);
      if (lane == 0 && t) atomicAdd(&s_tau, t);
      __syncthreads();
    }
    if (K >= 3) {
      for (int i = tid; i < d; i += NW * 32) tab_insert(tab, tb, list[i], i);
      __syncthreads();
      // Row i: N+(list[i]) ∩ N+(s).
      auto put = [&](int i, int j) {  // j, before i, is its neighbour
        if constexpr (MODE == MODE_SEQ) {
          atomicOr(&rows[(size_t)tri_off((uint32_t)i) + (j >> 5)], 1u << (j & 31));
        } else if constexpr (MODE == MODE_COUNT) {
          atomicOr(&rows[(size_t)i * W + (j >> 5)], 1u << (j & 31));
          atomicOr(&rows[(size_t)j * W + (i >> 5)], 1u << (i & 31));
        } else {
          const int ri = rank[i], rj = rank[j];
          const int lo = ri < rj ? ri : rj, hi = ri < rj ? rj : ri;
          atomicOr(&rows[(size_t)lo * W + (hi >> 5)], 1u << (hi & 31));
        }
      };
      induce_rows(
          a, list, d, tab, tb, wid, NW, lane,
          [&](int i, int w, bool hit) {
            if constexpr (MODE == MODE_SEQ) {
              const uint32_t m = __ballot_sync(KCL_FULL, hit);
              if (lane == 0) rows[(size_t)tri_off((uint32_t)i) + w] = m;
            } else if constexpr (MODE == MODE_COUNT) {
              const uint32_t m = __ballot_sync(KCL_FULL, hit);
              if (lane == 0 && m) atomicOr(&rows[(size_t)i * W + w], m);
              if (hit) atomicOr(&rows[(size_t)((w << 5) | lane) * W + (i >> 5)], 1u << (i & 31));
            } else if (hit) {
              put(i, (w << 5) | lane);
            }
          },
          put);
      __syncthreads();
    }
    if constexpr (MODE == MODE_SEQ) {
      if (a.shared_loads)
        seq_streams_shared<K, WPL>(next, d, rows, list, s, a.out, s_off, reinterpret_cast<uint32_t *>(acc), dl,
                                   lane, a.err);
      else
        seq_streams<K, WPL>(next, d, rows, base, dl, acc, rel, pair, lane, a.err);
      __syncthreads();
      for (int i = tid; i <= d; i += NW * 32) {
        const unsigned long long v = acc[i];
        if (v) {
          // shared loads: already in the load vector, stream by stream
          if (!a.shared_loads) atomicAdd(&a.out[i < d ? list[i] : s], v);
          acc[i] = 0;
        }
      }
    } else {
      const int tau = (MODE == MODE_ORDER) ? s_tau : 0;
      // COUNT, s's own share: the (k-1)-cliques of G_s.  A CTA that has the root
      // to itself divides the rows' total by k - 1; CTAs that split one sum the
      // cliques whose largest member is p, i.e. the (k-2)-cliques among p's
      // neighbours below it, a second walk.  Explicit lists take no share.
      // (Without the second walk: k = 4 count of RMAT-18 2.2 -> 1.7 ms.)
      const bool low = MODE == MODE_COUNT && a.active && !a.list_off;
      unsigned long long mine = 0;
      for (;;) {
        int p = 0;
        if (lane == 0) p = (int)(atomicAdd(next, 1u) & kTaskMask);
        p = __shfl_sync(KCL_FULL, p, 0);
        if (p >= d) break;
        const Bits<WPL> P = load_row<WPL>(rows, p, W, lane);
        uint64_t c = 0;
        uint64_t c_low = 0;
        if constexpr (K == 4 && WPL == 1 && ROWS_IN_SMEM) {
          c = __reduce_add_sync(KCL_FULL, edges_in<MODE == MODE_COUNT>(P, rows, W, lane, cbuf));
          if (MODE == MODE_COUNT && low)
            c_low = __reduce_add_sync(KCL_FULL, edges_in<true>(band(P, below_mask<WPL>(p, lane)), rows, W, lane, cbuf));
        } else if constexpr (K == 5 && WPL == 1 && ROWS_IN_SMEM) {
          // at most C(1023, 3) triangles: 32 bits
          c = __reduce_add_sync(KCL_FULL, triangles_in<MODE == MODE_COUNT>(P, rows, W, lane, cbuf));
          if (MODE == MODE_COUNT && low)
            c_low =
                __reduce_add_sync(KCL_FULL, triangles_in<true>(band(P, below_mask<WPL>(p, lane)), rows, W, lane, cbuf));
        } else {
          c = warp_sum(cnt_warp<K - 2, MODE == MODE_COUNT, WPL>(P, rows, W, lane));
          if (MODE == MODE_COUNT && low)
            c_low = warp_sum(cnt_warp<K - 2, true, WPL>(band(P, below_mask<WPL>(p, lane)), rows, W, lane));
        }
        if (lane == 0) {
          if (MODE == MODE_COUNT) {
            if (a.list_off) a.pair_out[o + p] = (unsigned long long)c;
            else if (c) atomicAdd(&a.out[list[p]], (unsigned long long)c);
            mine += low ? c_low : c;
          } else if (p < tau) {
            if (c) atomicAdd(&a.out[list[inv[p]]], (unsigned long long)c);
          } else {
            mine += c;
          }
        }
      }
      if (lane == 0 && mine) shared_add(&s_sum, mine);
      __syncthreads();
      if (tid == 0 && s_sum && !(MODE == MODE_COUNT && a.list_off)) {
        const unsigned long long own = MODE == MODE_COUNT && !low ? s_sum / (unsigned long long)(K - 1) : s_sum;
        atomicAdd(&a.out[s], own);
        if constexpr (IDENT && MODE == MODE_COUNT) atomicAdd(a.total, own);
      }
    }
    if (tid == 0 && a.active) a.active[blockIdx.x] = 0;
    __syncthreads();
  }
}

}  // namespace dev

// Per-kernel launch settings, computed once per (device, kernel, dynamic
// shared memory size): the opt-in shared-memory attribute (a per-device
// setting: cudaFuncSetAttribute applies to the current device only) and the
// number of CTAs one SM holds.  Launches then cost no runtime queries.
constexpr int kMaxDevices = 64;
struct LaunchCache {
  std::mutex mu;
  int attr_bytes[kMaxDevices];
  size_t occ_smem[64];  // fixed storage: launching never touches the heap
  int occ_dev[64];
  int occ_threads[64];
  int occ_ctas[64];
  int nocc = 0;
  // Seq tiers M / L: chosen warps per CTA by (device, out-degree bound, requested width).
  uint32_t nw_dmax[32];
  int nw_dev[32], nw_req[32], nw_val[32];
  int nnw = 0;
  LaunchCache() {
    for (int i = 0; i < kMaxDevices; ++i) attr_bytes[i] = -1;
  }
};

static inline int current_device() {
  int d = 0;
  if (cudaGetDevice(&d) != cudaSuccess || d < 0 || d >= kMaxDevices) d = 0;
  return d;
}

template <typename Fn>
static cudaError_t prepare(Fn fn, LaunchCache &lc, int threads, size_t smem, int *per_sm) {
  const int dev = current_device();
  std::lock_guard<std::mutex> g(lc.mu);
  if ((int)smem > lc.attr_bytes[dev]) {
    cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    lc.attr_bytes[dev] = (int)smem;
  }
  for (int i = 0; i < lc.nocc; ++i)
    if (lc.occ_dev[i] == dev && lc.occ_smem[i] == smem && lc.occ_threads[i] == threads) {
      *per_sm = lc.occ_ctas[i];
      return cudaSuccess;
    }
  int nb = 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, fn, threads, smem) != cudaSuccess || nb < 1) nb = 1;
  if (lc.nocc < 64) {
    lc.occ_dev[lc.nocc] = dev;
    lc.occ_smem[lc.nocc] = smem;
    lc.occ_threads[lc.nocc] = threads;
    lc.occ_ctas[lc.nocc] = nb;
    ++lc.nocc;
  }
  *per_sm = nb;
  return cudaSuccess;
}

// Warps per CTA of a tier M / L launch: `req` when nonzero, else the width
// that keeps the most warps resident per SM at this out-degree bound (ties:
// the narrower, i.e. more CTAs).  Seq: 8..24 in steps of 4, and on request 2
// or 4 (many small CTAs for groups of small roots, where a root has few root
// edges to share out); the counting kernels: 8..32 in steps of 8.
template <int MODE, int K, typename Fn>
static cudaError_t pick_warps(Fn fn, LaunchCache &lc, uint32_t dmax, bool rows_in_smem, int req, int *nw) {
  using namespace dev;
  constexpr int hi = warps_m<MODE, K>(), step = MODE == MODE_SEQ ? 4 : 8;
  const int lo = (MODE == MODE_SEQ && (req == 2 || req == 4)) ? req : 8;
  const int dev = current_device();
  {
    std::lock_guard<std::mutex> g(lc.mu);
    for (int i = 0; i < lc.nnw; ++i)
      if (lc.nw_dev[i] == dev && lc.nw_dmax[i] == dmax && lc.nw_req[i] == req) {
        *nw = lc.nw_val[i];
        return cudaSuccess;
      }
  }
  int best = 0, best_warps = -1;
  for (int w = lo; w <= hi; w = w < 8 ? w * 2 : w + step) {
    const size_t sm = layout_m(MODE, K, dmax, w, rows_in_smem).total;
    if (sm > 227 * 1024) continue;
    if (req > 0) {  // the requested width, or the widest below it that fits
      if (w <= req) best = w;
      continue;
    }
    int per_sm = 0;
    cudaError_t e = prepare(fn, lc, w * 32, sm, &per_sm);
    if (e != cudaSuccess) return e;
    if (per_sm * w > best_warps) { best_warps = per_sm * w; best = w; }
  }
  if (best == 0) best = lo;
  std::lock_guard<std::mutex> g(lc.mu);
  if (lc.nnw < 32) {
    lc.nw_dev[lc.nnw] = dev;
    lc.nw_dmax[lc.nnw] = dmax;
    lc.nw_req[lc.nnw] = req;
    lc.nw_val[lc.nnw] = best;
    ++lc.nnw;
  }
  *nw = best;
  return cudaSuccess;
}

// Persistent grid: as many CTAs as are resident at once.  Tier S needs no
// more warps than roots; tiers M and L keep every resident CTA, because a CTA
// without a root of its own steals sub-tasks from the unfinished roots.
static int persistent_grid(int per_sm, const TierLaunch &t, int roots_per_cta, bool steals) {
  long long g = (long long)per_sm * t.num_sms;
  if (!steals) {
    const long long need = ((long long)t.num_roots + roots_per_cta - 1) / roots_per_cta;
    if (need < g) g = need;
  }
  if (t.max_grid > 0 && g > t.max_grid) g = t.max_grid;
  if (steals && g > (long long)kActiveSlots) g = kActiveSlots;  // one registry slot per CTA
  return (int)(g < 1 ? 1 : g);
}

template <int MODE, int K>
cudaError_t launch_tier(const TierLaunch &t, dev::PassArgs a, cudaStream_t st) {
  using namespace dev;
  a.roots = t.roots;
  a.num_roots = t.num_roots;
  a.dmax = t.dmax;
  a.work = t.work;
  a.task_next = t.task_next;
  a.active = t.active;
  if (t.num_roots == 0) return cudaSuccess;
  int per_sm = 1;
  if (t.tier == 0) {
    static LaunchCache lc;
    const size_t sm = sizeof(SmemS<MODE>) * kWarpsS;
    auto fn = tier_s_kernel<MODE, K>;
    cudaError_t e = prepare(fn, lc, kWarpsS * 32, sm, &per_sm);
    if (e != cudaSuccess) return e;
    fn<<<persistent_grid(per_sm, t, kWarpsS, false), kWarpsS * 32, sm, st>>>(a);
    return cudaGetLastError();
  }
  if (t.tier == 1) {
    static LaunchCache lc;
    auto fn = tier_m_kernel<MODE, K, 1, true>;
    int nw = kWarpsM;
    cudaError_t e = pick_warps<MODE, K>(fn, lc, t.dmax, true, t.warps, &nw);
    if (e != cudaSuccess) return e;
    const size_t sm = layout_m(MODE, K, t.dmax, nw, true).total;
    e = prepare(fn, lc, nw * 32, sm, &per_sm);
    if (e != cudaSuccess) return e;
    // Shared loads: every stream in flight is blind to the others, so that too
    // large a share of a pass at once costs passes.  A launch takes at most a
    // 32nd of the root edges, but 24 warps an SM at least (20 of width 20, 16 of
    // width 16); the groups of a pass may run side by side, so the pass as a
    // whole can hold more.  Passes to a certified 1 % gap (what fits, 24 warps,
    // this): planted RMAT-13 at k = 5 92..101, 83, 83; planted RMAT-15 at k = 4
    // 45 with 24 warps, 35 so; 60,000 vertices with communities 16 and 9, and a
    // pass takes 475 and 385 us.  A planted RMAT-12 at k = 3 has its densest set
    // first after 64 passes in 308 of 360 runs with what fits, in 336 so (in 208
    // of 300 when each run is certified), and its pass takes 129 and 96 us.
    if (MODE == MODE_SEQ && a.shared_loads) {
      const uint64_t share = std::min<uint64_t>(t.streams / (32 * (uint64_t)t.num_sms), 64);
      per_sm = std::min(per_sm, std::max(1, (int)std::max<uint64_t>(share, 24) / nw));
    }
    fn<<<persistent_grid(per_sm, t, 1, t.active != nullptr), nw * 32, sm, st>>>(a);
    return cudaGetLastError();
  }
  static LaunchCache lc;
  auto fn = tier_m_kernel<MODE, K, 2, false>;
  int nw = kWarpsM;
  cudaError_t e = pick_warps<MODE, K>(fn, lc, t.dmax, false, t.warps, &nw);
  if (e != cudaSuccess) return e;
  const size_t sm = layout_m(MODE, K, t.dmax, nw, false).total;
  e = prepare(fn, lc, nw * 32, sm, &per_sm);
  if (e != cudaSuccess) return e;
  fn<<<persistent_grid(per_sm, t, 1, t.active != nullptr), nw * 32, sm, st>>>(a);
  return cudaGetLastError();
}

// The kernels of MODE for k in [LO, HI].
template <int MODE, int LO = 2, int HI = 8>
cudaError_t launch_mode(int k, const TierLaunch &t, dev::PassArgs a, cudaStream_t st) {
  if constexpr (LO > HI) {
    return cudaErrorInvalidValue;
  } else if constexpr (LO < 3 && MODE != dev::MODE_ORDER) {
    return launch_mode<MODE, 3, HI>(k, t, a, st);
  } else {
    return k == LO ? launch_tier<MODE, LO>(t, a, st) : launch_mode<MODE, LO + 1, HI>(k, t, a, st);
  }
}

}  // namespace kclpp
