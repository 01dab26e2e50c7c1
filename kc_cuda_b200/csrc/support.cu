// Stage (d): support (triangles through each edge) of the working graph.
//
// Dense mode (bitsets): the product of the rows on the tensor cores where the
// graph is dense enough for it (support_products), else a popcount per edge.
//
// List mode: the edges whose ends both have at most kFilterDeg neighbours are
// counted from the triangles' lowest vertices (k_support_filter, a warp per
// vertex).  The others are counted from their higher-degree end, with no
// atomics on the counts: a block owns a vertex v at a time, marks N(v) in a
// shared-memory bitmap over the subgraph's vertex ids, and for every lower
// neighbour u (new id < v, so deg(u) <= deg(v)) a warp scans N(u) against the
// bitmap; the popcount is |N(u) n N(v)|, written to the edge (u, v).  Blocks
// are persistent and take vertices from the highest degree down through an
// atomic cursor (k_support_bitmap).
//
// The reference counts triangles on the degree-oriented graph with a
// warp-per-vertex merge and scatters 2 per triangle to all three edges with
// atomics (tricount_direct, src/kc.cu:505-651); its support is twice this.
//
// Larger vertices of a graph whose vertex count exceeds the bitmap limit use
// k_support_search: warp per edge, lanes binary-search the shorter row in the
// longer one.
#include <algorithm>

#include <vector>

#include "compact.cuh"
#include "dense.cuh"
#include "stages.h"
#include "subgraph.h"
#include "support_mma.h"

namespace kt {
namespace {

constexpr unsigned kSupThreads = 256;
constexpr unsigned kSupThreadsWide = 1024;  // bitmap kernel when its bitmap limits blocks per SM

// Edges whose ends have at most kFilterDeg neighbours: every triangle u < v <
// w with such u and v is found once, from its lowest vertex u, by scanning the
// upper neighbours of each upper neighbour v of u against those of u; it adds
// one to (u, v), and to (u, w) and (v, w) where w is such a vertex too (the
// edges to longer rows are counted by the kernels below).  Scanning upper parts
// only reads a third of what the whole rows of the smaller ends hold on an
// Erdos-Renyi graph.  Sup must be zero before.
//
// A warp owns u.  Its upper neighbours are kept in a shared-memory table with
// one slot per hash value, which holds the neighbour that hashes there (and
// its place in the row) or, where several do, a mark that sends the lookup to
// the row.  Four rows are streamed side by side, 8 lanes each and 8 entries
// per lane in flight; an entry costs one coalesced load, a hash, a
// shared-memory load and two compares, and the kernel is bound by issuing
// those.  The line at 256 neighbours keeps the marked slots under 4 %.
// Measured against a block and a bitmap per vertex: Erdos-Renyi, 250,007
// vertices, 7.9M edges 2.49 -> 0.58 ms; 10^6 vertices, 64M edges 34.5 -> 9.3 ms
// (whole rows and a table of bits instead took 0.96 and 19.0 ms).
constexpr uint32_t kFilterDeg = 256;
constexpr uint32_t kFilterSlots = 1024;
constexpr uint32_t kSlotEmpty = 0xffffffffu, kSlotMany = 0xfffffffeu;  // no vertex has these ids

__device__ __forceinline__ uint32_t filter_slot(uint32_t w) { return (w * 0x9E3779B1u) >> 22; }
static_assert(kFilterSlots == 1u << (32 - 22), "filter_slot yields 10 bits");

__global__ void __launch_bounds__(kSupThreads) k_support_filter(uint32_t n, const uint64_t* __restrict__ off,
                                                                const uint32_t* __restrict__ adj,
                                                                const uint32_t* __restrict__ eid,
                                                                const uint64_t* __restrict__ up,
                                                                uint32_t* __restrict__ sup) {
  __shared__ uint32_t s_slot[kSupThreads / 32][kFilterSlots];
  __shared__ uint8_t s_place[kSupThreads / 32][kFilterSlots];
  uint32_t* slot = s_slot[warp_id()];
  uint8_t* place = s_place[warp_id()];
  const unsigned lane = lane_id();
  for (uint32_t i = lane; i < kFilterSlots; i += 32) slot[i] = kSlotEmpty;
  __syncwarp();
  const uint64_t warps = (uint64_t)gridDim.x * (blockDim.x >> 5);
  for (uint64_t u = (uint64_t)blockIdx.x * (blockDim.x >> 5) + warp_id(); u < n; u += warps) {
    const uint64_t uu = up[u], ue = off[u + 1];
    // A triangle needs two upper neighbours of u.
    if (ue - off[u] > kFilterDeg || ue - uu < 2) continue;
    const uint32_t d = (uint32_t)(ue - uu);
    const uint32_t* mine = adj + uu;
    for (uint32_t i = lane; i < d; i += 32) {
      const uint32_t w = mine[i], h = filter_slot(w);
      if (atomicCAS(&slot[h], kSlotEmpty, w) == kSlotEmpty)
        place[h] = (uint8_t)i;
      else
        slot[h] = kSlotMany;
    }
    __syncwarp();
    for (uint32_t c0 = 0; c0 < d; c0 += 32) {
      const uint32_t i = c0 + lane;
      uint64_t rb = 0;
      uint32_t len = 0;
      if (i < d) {
        const uint32_t v = mine[i];
        const uint64_t e = off[v + 1];
        rb = up[v];
        len = e - off[v] > kFilterDeg ? 0u : (uint32_t)(e - rb);
      }
      const uint32_t cn = min(32u, d - c0);
      for (uint32_t q = 0; q < cn; q += 4) {
        const uint32_t from = q + (lane >> 3);
        const uint64_t b = __shfl_sync(kFull, rb, from);
        const uint32_t l = __shfl_sync(kFull, len, from);
        uint32_t cnt = 0;
        const uint32_t* row = adj + b;
        for (uint32_t k = lane & 7; k < l; k += 64) {
          uint32_t w[8];
#pragma unroll
          for (uint32_t t = 0; t < 8; ++t) w[t] = k + 8 * t < l ? row[k + 8 * t] : (uint32_t)u;  // u is not above u
#pragma unroll
          for (uint32_t t = 0; t < 8; ++t) {
            const uint32_t h = filter_slot(w[t]);
            const uint32_t at = slot[h];
            if (at == w[t] || at == kSlotMany) {
              uint32_t p;
              if (at == kSlotMany) {
                uint32_t lo = 0, hi = d;
                while (lo < hi) {
                  const uint32_t mid = (lo + hi) >> 1;
                  if (mine[mid] < w[t])
                    lo = mid + 1;
                  else
                    hi = mid;
                }
                if (lo == d || mine[lo] != w[t]) continue;
                p = lo;
              } else {
                p = place[h];
              }
              ++cnt;
              if (off[w[t] + 1] - off[w[t]] <= kFilterDeg) {
                atomicAdd(&sup[eid[uu + p]], 1u);
                atomicAdd(&sup[eid[b + k + 8 * t]], 1u);
              }
            }
          }
        }
        __syncwarp();
#pragma unroll
        for (int o = 4; o > 0; o >>= 1) cnt += __shfl_xor_sync(kFull, cnt, o);
        if ((lane & 7) == 0 && cnt) atomicAdd(&sup[eid[uu + c0 + from]], cnt);
      }
    }
    __syncwarp();
    for (uint32_t i = lane; i < d; i += 32) slot[filter_slot(mine[i])] = kSlotEmpty;
    __syncwarp();
  }
}

// Vertices k_support_filter leaves out.
struct LongRow {
  const uint64_t* off;
  __device__ bool keep(uint64_t v) const { return off[v + 1] - off[v] > kFilterDeg; }
  __device__ uint32_t value(uint64_t v) const { return (uint32_t)v; }
};

// The n vertices of `list` (ascending).  Batched unions: the bitmap covers
// only v's own graph, bits indexed from vbase[v] (graphs are contiguous and no
// edge crosses graphs); `range` = most vertices of one graph.
__global__ void __launch_bounds__(kSupThreadsWide) k_support_bitmap(const uint32_t* __restrict__ list, uint32_t n,
                                                                const uint64_t* __restrict__ off,
                                                                const uint32_t* __restrict__ adj,
                                                                const uint32_t* __restrict__ eid,
                                                                const uint64_t* __restrict__ up,
                                                                uint32_t* __restrict__ sup,
                                                                unsigned long long* cursor,
                                                                const uint32_t* __restrict__ vbase, uint32_t range) {
  extern __shared__ uint32_t bits[];
  __shared__ uint32_t s_v;
  const uint32_t words = (range + 31) / 32;
  for (uint32_t i = threadIdx.x; i < words; i += blockDim.x) bits[i] = 0;
  __syncthreads();
  while (true) {
    if (threadIdx.x == 0) {
      const unsigned long long t = atomicAdd(cursor, 1ULL);
      s_v = t < n ? list[n - 1 - t] : 0xffffffffu;
    }
    __syncthreads();
    const uint32_t v = s_v;
    if (v == 0xffffffffu) break;
    const uint32_t base = vbase ? vbase[v] : 0u;
    const uint64_t vb = off[v], ve = off[v + 1], vu = up[v];
    for (uint64_t j = vb + threadIdx.x; j < ve; j += blockDim.x) {
      const uint32_t w = adj[j] - base;
      atomicOr(&bits[w >> 5], 1u << (w & 31));
    }
    __syncthreads();
    // Lower neighbours u of v: entries [vb, vu).
    for (uint64_t j = vb + warp_id(); j < vu; j += blockDim.x >> 5) {
      const uint32_t u = adj[j];
      const uint64_t ub = off[u], ue = off[u + 1];
      uint32_t cnt = 0;
      for (uint64_t q = ub + lane_id(); q < ue; q += 32) {
        const uint32_t w = adj[q] - base;
        cnt += (bits[w >> 5] >> (w & 31)) & 1u;
      }
      cnt = warp_sum(cnt);
      if (lane_id() == 0) sup[eid[j]] = cnt;
    }
    __syncthreads();
    for (uint64_t j = vb + threadIdx.x; j < ve; j += blockDim.x) {
      const uint32_t w = adj[j] - base;
      bits[w >> 5] = 0;
    }
    __syncthreads();
  }
}

// Position of x in sorted a[lo, hi), or hi.
__device__ __forceinline__ uint64_t find_sorted(const uint32_t* a, uint64_t lo, uint64_t hi, uint32_t x) {
  const uint64_t end = hi;
  while (lo < hi) {
    const uint64_t mid = (lo + hi) >> 1;
    if (a[mid] < x)
      lo = mid + 1;
    else
      hi = mid;
  }
  return (lo < end && a[lo] == x) ? lo : end;
}

// Edges whose larger end has more than kFilterDeg neighbours.
__global__ void k_support_search(uint64_t m, const uint64_t* __restrict__ ends, const uint64_t* __restrict__ off,
                                 const uint32_t* __restrict__ adj, uint32_t* __restrict__ sup) {
  const uint64_t warps = (uint64_t)gridDim.x * (blockDim.x >> 5);
  for (uint64_t e = (uint64_t)blockIdx.x * (blockDim.x >> 5) + warp_id(); e < m; e += warps) {
    const uint64_t k = ends[e];
    uint32_t a = (uint32_t)(k >> 32), b = (uint32_t)k;
    if (off[b + 1] - off[b] <= kFilterDeg) continue;  // the end with the larger id owns the edge
    if (off[a + 1] - off[a] > off[b + 1] - off[b]) {
      const uint32_t t = a;
      a = b;
      b = t;
    }
    const uint64_t ab = off[a], ae = off[a + 1], bb = off[b], be = off[b + 1];
    uint32_t cnt = 0;
    for (uint64_t q = ab + lane_id(); q < ae; q += 32) cnt += find_sorted(adj, bb, be, adj[q]) != be;
    cnt = warp_sum(cnt);
    if (lane_id() == 0) sup[e] = cnt;
  }
}

// Dense mode: row bitsets from the sorted rows.
__global__ void k_bits_build(uint32_t n, const uint64_t* __restrict__ off, const uint32_t* __restrict__ adj,
                             DenseRows R) {
  const uint64_t warps = (uint64_t)gridDim.x * (blockDim.x >> 5);
  for (uint64_t u = (uint64_t)blockIdx.x * (blockDim.x >> 5) + warp_id(); u < n; u += warps) {
    uint32_t* row = R.bits + R.off((uint32_t)u);
    for (uint64_t j = off[u] + lane_id(); j < off[u + 1]; j += 32) {
      const uint32_t v = R.col((uint32_t)u, adj[j]);
      atomicOr(&row[v >> 5], 1u << (v & 31));
    }
  }
}

// spre[w] = set bits of row u before its word w (warp per row).
__global__ void k_row_prefix(uint32_t n, DenseRows R, uint32_t* __restrict__ spre) {
  const uint64_t warps = (uint64_t)gridDim.x * (blockDim.x >> 5);
  for (uint64_t u = (uint64_t)blockIdx.x * (blockDim.x >> 5) + warp_id(); u < n; u += warps) {
    const uint64_t base = R.off((uint32_t)u);
    const uint32_t W = R.words((uint32_t)u);
    uint32_t run = 0;
    for (uint32_t i0 = 0; i0 < W; i0 += 32) {
      const uint32_t i = i0 + lane_id();
      const uint32_t pc = i < W ? __popc(R.bits[base + i]) : 0u;
      const uint32_t inc = warp_incl_scan(pc);
      if (i < W) spre[base + i] = run + inc - pc;
      run += __shfl_sync(kFull, inc, 31);
    }
  }
}

// Per-graph rows of a grouped union: graph g's rows hold gw[g] words and
// start at word gbase[g].
__global__ void k_group_rows(uint32_t n, const uint32_t* __restrict__ vgid, const uint32_t* __restrict__ vbase,
                             const uint64_t* __restrict__ gbase, const uint32_t* __restrict__ gw,
                             uint64_t* __restrict__ roff, uint32_t* __restrict__ rw) {
  for (uint64_t v = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; v < n; v += (uint64_t)gridDim.x * blockDim.x) {
    const uint32_t g = vgid[v];
    roff[v] = gbase[g] + (uint64_t)(v - vbase[v]) * gw[g];
    rw[v] = gw[g];
  }
}

// Warps take 32-edge groups from a cursor, so the groups in flight stay a
// narrow window of the tile-ordered list (a grid-stride loop lets warps drift
// apart, and the rows they read then no longer fit in L2).  `row_words`
// accumulates the row words read.
//
// Exact counts, up to NQ edges sharing row u per shared-memory read of it;
// four resident blocks per SM (what the rows' shared memory allows for the
// bench graph's cores) bound the registers to 64.
template <int NQ>
__global__ void __launch_bounds__(256, 4) k_dense_support(uint64_t m, const uint32_t* __restrict__ order,
                                                          const uint64_t* __restrict__ ends, DenseRows R,
                                                          uint32_t* __restrict__ sup,
                                                          unsigned long long* __restrict__ row_words,
                                                          unsigned long long* __restrict__ cursor) {
  extern __shared__ __align__(16) uint32_t dense_smem[];
  uint32_t* su = dense_smem + warp_id() * R.W;
  const uint64_t groups = (m + 31) / 32;
  unsigned long long wr = 0;  // row words this lane accounts for (lane 0)
  for (;;) {
    unsigned long long g = 0;
    if (lane_id() == 0) g = atomicAdd(cursor, 1ULL);
    g = __shfl_sync(kFull, g, 0);
    if (g >= groups) break;
    uint32_t e, s;
    bool ok;
    dense_group<NQ>(order, g * 32, m, ends, R, nullptr, su, e, s, ok, &wr);
    if (ok) sup[e] = s;
  }
  wr = warp_sum(wr);
  if (lane_id() == 0 && wr) atomicAdd(row_words, wr);
}

// Exact counts over rows of at most kShortRow words, from 8-entry groups (a
// warp works on eight edges at once).
__global__ void __launch_bounds__(256) k_dense_support_short(uint64_t m, const uint32_t* __restrict__ order,
                                                             const uint64_t* __restrict__ ends, DenseRows R,
                                                             uint32_t* __restrict__ sup,
                                                             unsigned long long* __restrict__ row_words) {
  const uint64_t warps = (uint64_t)gridDim.x * (blockDim.x >> 5);
  const uint32_t size = m / warps >= 32 ? 32u : 8u;
  unsigned long long wr = 0;
  for (uint64_t g = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; g * size < m; g += warps) {
    uint32_t e, s;
    bool ok;
    dense_group_short(order, g * size, min(m, (g + 1) * size), ends, R, nullptr, size / 4, e, s, ok, &wr);
    if (ok) sup[e] = s;
  }
  wr = warp_sum(wr);
  if (lane_id() == 0 && wr) atomicAdd(row_words, wr);
}

// Capped counts (search phase): threshold `cap`, or gcap[vgid[u]] per graph
// of a grouped union.
__global__ void __launch_bounds__(256) k_dense_support_capped(uint64_t m, const uint32_t* __restrict__ order,
                                                              const uint64_t* __restrict__ ends, DenseRows R,
                                                              uint32_t cap, const uint32_t* __restrict__ gcap,
                                                              const uint32_t* __restrict__ vgid,
                                                              uint32_t* __restrict__ sup,
                                                              unsigned long long* __restrict__ row_words,
                                                              unsigned long long* __restrict__ cursor) {
  extern __shared__ __align__(16) uint32_t dense_smem[];
  uint32_t* su = dense_smem + warp_id() * R.W;
  const uint64_t groups = (m + 31) / 32;
  unsigned long long wr = 0;  // row words this lane accounts for (lanes 0 and 16)
  for (;;) {
    unsigned long long g = 0;
    if (lane_id() == 0) g = atomicAdd(cursor, 1ULL);
    g = __shfl_sync(kFull, g, 0);
    if (g >= groups) break;
    uint32_t e, s;
    bool ok;
    dense_group_capped(order, g * 32, m, ends, R, cap, su, e, s, ok, &wr, gcap, vgid);
    if (ok) sup[e] = s;
  }
  wr = warp_sum(wr);
  if (lane_id() == 0 && wr) atomicAdd(row_words, wr);
}

// The entries of a tile-ordered list whose graphs are not flagged.
struct Uncounted {
  const uint32_t* order;
  const uint64_t* ends;
  const uint32_t* vgid;
  const uint8_t* counted;
  __device__ bool keep(uint64_t i) const { return !counted[vgid[(uint32_t)(ends[order[i]] >> 32)]]; }
  __device__ uint32_t value(uint64_t i) const { return order[i]; }
};

// Tile keys: (u >> tb) << 16 | (v >> tb), stable-sorted with the edge ids.
__global__ void k_tile_keys(uint64_t m, const uint64_t* __restrict__ ends, uint32_t tb, uint64_t* __restrict__ keys,
                            uint32_t* __restrict__ ids) {
  for (uint64_t e = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; e < m; e += (uint64_t)gridDim.x * blockDim.x) {
    const uint64_t k = ends[e];
    keys[e] = ((k >> (32 + tb)) << 16) | (((uint32_t)k) >> tb);
    ids[e] = (uint32_t)e;
  }
}

// Grid of the resident blocks of `kernel` with the rows' shared memory.
unsigned dense_grid(Ctx* c, const void* kernel, uint64_t m, size_t smem) {
  allow_max_dynamic_smem(kernel);
  int per_sm = 0;
  KT_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, 256, smem));
  return grid_for((m + 31) / 32 * 32, 256, std::max(1, per_sm) * c->num_sms);
}

template <int NQ>
void launch_exact(Ctx* c, const Sub& s, const uint32_t* order, uint64_t m, uint32_t* sup, unsigned long long* row_words,
                  unsigned long long* cursor) {
  const size_t smem = dense_smem_bytes(s.W, 256);
  const unsigned grid = dense_grid(c, (const void*)k_dense_support<NQ>, m, smem);
  k_dense_support<NQ><<<grid, 256, smem, c->stream>>>(m, order, s.ends.as<uint64_t>(),
                                                      dense_rows(s), sup, row_words, cursor);
  KT_LAUNCHED(c);
}

// Exact counts: option support_rows (1, 2 or 4) edges sharing row u per
// shared-memory read of it.  Capped counts: two edges sharing row u side by
// side, one per half of the warp.
void launch_dense_support(Ctx* c, const Sub& s, const uint32_t* order, uint64_t m, uint32_t* sup, bool capped,
                          uint32_t cap, const uint32_t* gcap,
                          unsigned long long* row_words, unsigned long long* cursor) {
  if (s.W <= kShortRow) {  // (exact also where a cap is given: there is little to abandon)
    k_dense_support_short<<<grid_for((m + 7) / 8 * 32, 256, c->num_sms * 8), 256, 0, c->stream>>>(
        m, order, s.ends.as<uint64_t>(), dense_rows(s), sup, row_words);
    KT_LAUNCHED(c);
  } else if (capped) {
    const size_t smem = dense_smem_bytes(s.W, 256);
    const unsigned grid = dense_grid(c, (const void*)k_dense_support_capped, m, smem);
    k_dense_support_capped<<<grid, 256, smem, c->stream>>>(m, order, s.ends.as<uint64_t>(),
                                                           dense_rows(s), cap, gcap,
                                                           gcap ? s.vgid.as<uint32_t>() : nullptr, sup, row_words,
                                                           cursor);
    KT_LAUNCHED(c);
  } else if (c->opt.support_rows <= 1) {
    launch_exact<1>(c, s, order, m, sup, row_words, cursor);
  } else if (c->opt.support_rows == 2) {
    launch_exact<2>(c, s, order, m, sup, row_words, cursor);
  } else {
    launch_exact<4>(c, s, order, m, sup, row_words, cursor);
  }
}

// Algorithmic bytes of a merge-based support count over the degree-oriented
// graph: 4 * sum over oriented edges (u -> v) of (d+(u) + d+(v)).
__global__ void k_support_alg(uint64_t m, const uint64_t* __restrict__ ends, const uint64_t* __restrict__ off,
                              const uint64_t* __restrict__ up, unsigned long long* out) {
  uint64_t s = 0;
  for (uint64_t e = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; e < m; e += (uint64_t)gridDim.x * blockDim.x) {
    const uint64_t k = ends[e];
    const uint32_t u = (uint32_t)(k >> 32), v = (uint32_t)k;
    s += (off[u + 1] - up[u]) + (off[v + 1] - up[v]);
  }
  s = warp_sum(s);
  if (lane_id() == 0 && s) atomicAdd(out, (unsigned long long)s);
}

// hist[min(sup, cap)] += 1.  Supports of a core crowd into few bins, so a block
// counts the first kHistBins in shared memory and adds them up at its end
// (10.5M edges, 1,686 bins: 0.61 ms with an atomic per distinct bin of a warp,
// below 0.03 now).
__global__ void __launch_bounds__(256) k_sup_hist(const uint32_t* __restrict__ sup, uint64_t m, uint32_t cap,
                                                  unsigned long long* __restrict__ hist) {
  __shared__ uint32_t bins[kHistBins];
  const uint32_t have = min(cap + 1, kHistBins);
  for (uint32_t b = threadIdx.x; b < have; b += blockDim.x) bins[b] = 0;
  __syncthreads();
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < m; i += (uint64_t)gridDim.x * blockDim.x) {
    const uint32_t b = min(sup[i], cap);
    if (b < kHistBins)
      atomicAdd(&bins[b], 1u);
    else
      atomicAdd(&hist[b], 1ULL);
  }
  __syncthreads();
  for (uint32_t b = threadIdx.x; b < have; b += blockDim.x)
    if (bins[b]) atomicAdd(&hist[b], (unsigned long long)bins[b]);
}

}  // namespace

uint32_t support_bound(Ctx* c, const uint32_t* sup, uint64_t m, uint32_t cap) {
  if (m == 0 || cap < 3) return 0;
  DBuf hist(c, ((uint64_t)cap + 1) * 8);
  zero(c, hist.get(), hist.bytes());
  k_sup_hist<<<grid_for(m, 256, c->num_sms * 4), 256, 0, c->stream>>>(sup, m, cap,
                                                                      hist.as<unsigned long long>());
  KT_LAUNCHED(c);
  std::vector<unsigned long long> h(cap + 1);
  copy_d2h(c, h.data(), hist.get(), h.size() * sizeof(unsigned long long));
  // at_least = edges with support >= t-2, accumulated while t descends.
  unsigned long long at_least = h[cap] + h[cap - 1];
  for (uint32_t t = cap; t >= 3; --t) {
    at_least += h[t - 2];
    if (at_least >= (unsigned long long)t * (t - 1) / 2) return t;
  }
  return 0;
}

bool build_bits(Ctx* c, Sub& s) {
  s.W = 0;
  s.bits.release();
  s.sbits.release();
  s.spre.release();
  s.roff.release();
  s.rw.release();
  s.bit_words = 0;
  if (s.n == 0 || s.m == 0) return false;
  // Rows: one block of bitsets per graph for a grouped union (every graph
  // within the vertex limit), else one block for the whole graph.
  const bool grouped = s.vgid.get() != nullptr && !s.group_n.empty();
  uint32_t W = 0;
  uint64_t words = 0;
  std::vector<uint64_t> gbase;
  std::vector<uint32_t> gw;
  if (grouped) {
    if ((int64_t)s.max_group > c->opt.dense_max_n) return false;
    gbase.resize(s.group_n.size());
    gw.resize(s.group_n.size());
    for (size_t g = 0; g < s.group_n.size(); ++g) {
      gbase[g] = words;
      gw[g] = ((s.group_n[g] + 31) / 32 + 3) & ~3u;  // rows of whole 16-byte vectors
      words += (uint64_t)s.group_n[g] * gw[g];
      W = std::max(W, gw[g]);
    }
  } else {
    if ((int64_t)s.n > c->opt.dense_max_n) return false;
    W = ((s.n + 31) / 32 + 3) & ~3u;  // rows of whole 16-byte vectors
    words = (uint64_t)s.n * W;
  }
  // Dense enough: adjacency entries * fill >= words of all rows.
  if (2.0 * (double)s.m * (double)c->opt.dense_min_fill < (double)words) return false;
  const uint64_t bytes = words * 4;
  if (c->budget && c->in_use + 2 * bytes > c->budget) return false;
  s.bits.alloc(c, bytes);
  zero(c, s.bits.get(), bytes);
  if (grouped) {
    const uint32_t G = (uint32_t)gw.size();
    DBuf dgb(c, G * 8ull), dgw(c, G * 4ull);
    copy_h2d(c, dgb.get(), gbase.data(), G * 8ull);
    copy_h2d(c, dgw.get(), gw.data(), G * 4ull);
    s.roff.alloc(c, (uint64_t)s.n * 8);
    s.rw.alloc(c, (uint64_t)s.n * 4);
    k_group_rows<<<grid_for(s.n, 256, c->num_sms * 16), 256, 0, c->stream>>>(
        s.n, s.vgid.as<uint32_t>(), s.vbase.as<uint32_t>(), dgb.as<uint64_t>(), dgw.as<uint32_t>(),
        s.roff.as<uint64_t>(), s.rw.as<uint32_t>());
    KT_LAUNCHED(c);
  }
  s.W = W;
  s.bit_words = words;
  k_bits_build<<<grid_for((uint64_t)s.n * 32, 256, c->num_sms * 16), 256, 0, c->stream>>>(
      s.n, s.off.as<uint64_t>(), s.adj.as<uint32_t>(), dense_rows(s));
  KT_LAUNCHED(c);
  // The rows as built and their per-word prefix counts (positions of
  // neighbours for the peel), when two more copies fit the budget.
  s.sbits.release();
  s.spre.release();
  if (!c->budget || c->in_use + 3 * bytes <= c->budget) {
    s.sbits.alloc(c, bytes);
    s.spre.alloc(c, bytes);
    KT_CUDA(cudaMemcpyAsync(s.sbits.get(), s.bits.get(), bytes, cudaMemcpyDeviceToDevice, c->stream));
    k_row_prefix<<<grid_for((uint64_t)s.n * 32, 256, c->num_sms * 16), 256, 0, c->stream>>>(
        s.n, dense_rows(s), s.spre.as<uint32_t>());
    KT_LAUNCHED(c);
  }
  // Tile order: blocks of 2^tb vertices, two blocks' bitsets within ~48 MB.
  uint32_t tb = 16;
  const uint64_t tile_bytes = (uint64_t)std::max<int64_t>(1, c->opt.dense_tile_mb) << 20;
  while (tb > 6 && 2ull * (1ull << tb) * W * 4 > tile_bytes) --tb;
  s.tile_bits = tb;
  s.order.alloc(c, s.m * sizeof(uint32_t));
  DBuf keys(c, s.m * sizeof(uint64_t));
  k_tile_keys<<<grid_for(s.m, 256, c->num_sms * 16), 256, 0, c->stream>>>(s.m, s.ends.as<uint64_t>(), tb,
                                                                            keys.as<uint64_t>(),
                                                                            s.order.as<uint32_t>());
  KT_LAUNCHED(c);
  const int blocks_bits = bits_for(((uint64_t)(s.n - 1) >> tb) + 1);
  radix_sort_u64(c, keys.as<uint64_t>(), s.order.as<uint32_t>(), s.m, {{0, blocks_bits}, {16, 16 + blocks_bits}});
  return true;
}

// List mode: k_support_filter, then the edges whose larger end it left out.
static void support_lists(Ctx* c, const Sub& s, uint32_t* sup) {
  const uint32_t range = s.vbase.get() ? s.max_group : s.n;
  const bool bitmap = (int64_t)range <= c->opt.support_bitmap_max_n;
  const size_t smem = ((range + 31) / 32) * sizeof(uint32_t);
  // Large bitmaps leave room for few blocks per SM: then wider blocks.
  const unsigned threads = smem > 24 * 1024 ? kSupThreadsWide : kSupThreads;
  int per_sm = 0;
  if (bitmap) {
    if (smem > 48 * 1024) allow_max_dynamic_smem((const void*)k_support_bitmap);
    KT_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_support_bitmap, threads, smem));
    if (per_sm < 1) throw Error(KT_ERR_LIMIT, "support: bitmap does not fit in shared memory");
  }
  zero(c, sup, s.m * sizeof(uint32_t));
  k_support_filter<<<grid_for((uint64_t)s.n * 32, kSupThreads, c->num_sms * 8), kSupThreads, 0, c->stream>>>(
      s.n, s.off.as<uint64_t>(), s.adj.as<uint32_t>(), s.eid.as<uint32_t>(), s.up.as<uint64_t>(), sup);
  KT_LAUNCHED(c);
  // (max_deg is the last vertex's degree, the largest of one graph only.)
  if (!s.vbase.get() && s.max_deg <= kFilterDeg) return;
  if (!bitmap) {
    k_support_search<<<grid_for(s.m * 32, 256, c->num_sms * 16), 256, 0, c->stream>>>(
        s.m, s.ends.as<uint64_t>(), s.off.as<uint64_t>(), s.adj.as<uint32_t>(), sup);
    KT_LAUNCHED(c);
    return;
  }
  DBuf list(c, (uint64_t)s.n * sizeof(uint32_t));
  const uint64_t nl = compact(c, s.n, LongRow{s.off.as<uint64_t>()}, list.as<uint32_t>());
  if (!nl) return;
  lower_ids(c, s);
  DBuf cur(c, 8);
  zero(c, cur.get(), 8);
  const unsigned grid = (unsigned)std::min<uint64_t>((uint64_t)per_sm * c->num_sms, nl);
  k_support_bitmap<<<grid, threads, smem, c->stream>>>(
      list.as<uint32_t>(), (uint32_t)nl, s.off.as<uint64_t>(), s.adj.as<uint32_t>(), s.eid.as<uint32_t>(),
      s.up.as<uint64_t>(), sup, cur.as<unsigned long long>(), s.vbase.get() ? s.vbase.as<uint32_t>() : nullptr, range);
  KT_LAUNCHED(c);
}

void edge_support(Ctx* c, const Sub& s, uint32_t* sup, uint32_t cap, const uint32_t* gcap) {
  if (s.m == 0) return;
  // acc[0]: merge-model list entries, acc[1]: dense row words read, acc[2]:
  // the dense kernel's group cursor.
  DBuf acc(c, 24);
  zero(c, acc.get(), 24);
  cudaEvent_t e0;
  if (c->opt.verbose) KT_CUDA(cudaEventRecord(c->ev[2], c->stream));
  c->timer.begin(c->stream, &c->stats.ms_support_kernel, &e0);
  uint64_t product_words = 0;
  const uint32_t* order = s.W ? s.order.as<uint32_t>() : nullptr;
  uint64_t left = s.m;  // edges of `order` that the products leave
  DBuf rest;
  std::vector<uint8_t> counted;
  const bool products = support_products(c, s, sup, cap || (gcap && s.vgid.get()), counted, &product_words);
  if (products) {
    left = 0;
    if (!counted.empty() && std::find(counted.begin(), counted.end(), 0) != counted.end()) {
      DBuf flags(c, counted.size());
      copy_h2d(c, flags.get(), counted.data(), counted.size());
      rest.alloc(c, s.m * sizeof(uint32_t));
      left = compact(c, s.m, Uncounted{order, s.ends.as<uint64_t>(), s.vgid.as<uint32_t>(), flags.as<uint8_t>()},
                     rest.as<uint32_t>());
      order = rest.as<uint32_t>();
    }
  }
  if (!left) {
  } else if (s.W) {
    unsigned long long* a = acc.as<unsigned long long>();
    const bool capped = cap || (gcap && s.vgid.get());
    launch_dense_support(c, s, order, left, sup, capped, cap, s.vgid.get() ? gcap : nullptr, a + 1, a + 2);
  } else {
    support_lists(c, s, sup);
  }
  c->timer.end(c->stream, e0, &c->stats.ms_support_kernel);
  if (c->opt.verbose) KT_CUDA(cudaEventRecord(c->ev[3], c->stream));
  c->stats.support_launches++;
  // Algorithmic bytes (outside the timed span): the merge model, and the
  // bytes the kernel that ran moved.
  k_support_alg<<<grid_for(s.m, 256, c->num_sms * 8), 256, 0, c->stream>>>(s.m, s.ends.as<uint64_t>(),
                                                                             s.off.as<uint64_t>(),
                                                                             s.up.as<uint64_t>(),
                                                                             acc.as<unsigned long long>());
  KT_LAUNCHED(c);
  uint64_t h[2];
  read_checked(c, h, acc.get(), 16, "support");
  h[1] += product_words;
  const uint64_t merge = 4 * h[0] + 4 * s.m + 8 * ((uint64_t)s.n + 1);
  c->stats.support_bytes += merge;
  c->stats.support_row_words += h[1];
  // Dense: row words, plus per edge its list entry (4), ends (8) and result (4).
  c->stats.support_kernel_bytes += s.W ? 4 * h[1] + 16 * s.m : merge;
  KT_LOG(c, "kt: support (%s) on %u vertices (widest group %u), %llu edges: %llu row words, %.3f ms\n",
         products ? "products" : s.W ? (cap || (gcap && s.vgid.get()) ? "dense capped" : "dense") : "list", s.n,
         s.vbase.get() ? s.max_group : s.n, (unsigned long long)s.m, (unsigned long long)h[1],
         c->opt.verbose ? event_ms(c->ev[2], c->ev[3]) : 0.0);
}

}  // namespace kt
