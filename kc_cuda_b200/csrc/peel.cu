// Stage (e): truss peeling of the working graph.
//
// Levels: at truss level t every alive edge with support < t-2 is removed,
// round by round, until none is left (a cascade); the alive edges then form
// the t-truss.  If edges remain, their minimum support s makes them an
// (s+2)-truss, which is recorded, and the next level is t = s+3.  The last
// recorded level when no edge is left is kmax.
//
// Rounds: the frontier edges of round r carry state r; deleted edges keep
// their round, alive edges kAlive.  Without bitsets, the entries w of the
// shorter row of a frontier edge (x, y) are looked up as edges to its other
// end in a hash table of the edges (list_round).  With bitsets, a warp takes a
// frontier edge and ANDs the two rows, or where the sorted rows are shorter
// (and in list mode without a table) merges them: 32-wide tiles of both rows
// are compared with a 5-step shuffle search, and whichever tile ends lower is
// retired (both when the ends tie), so every common neighbour is met exactly
// once; when one row is more than peel_search_ratio (16) times longer the lanes
// binary-search the long row instead.  A common w closes the triangle {e, a, b};
// it is skipped if a or b was deleted in an earlier round.  Each surviving side edge loses one
// triangle, decremented by exactly one frontier edge of the triangle (the
// one with the smallest id among those in this round); an edge whose support
// steps from t-2 to t-3 joins the next frontier, so each edge enters a
// frontier once.
//
// Levels run in one cooperative launch (k_levels): rounds are separated by the
// bounded grid barrier, the alive list is compacted and the next level chosen
// on the device, and the launch ends when the graph is empty or the host has
// something to do (a smaller graph to build, a bisection to start).
//
// Jumps: without per-edge trussness output, the first level may be a guess
// well above the lower bound (one cascade removes everything below it).  The
// support/state arrays are snapshotted first; a guess that empties the graph
// is undone and halved toward the last good level.
//
// The reference keeps doubled supports and subtracts 2 - [m1==st] - [m2==st]
// from both side edges (src/kc.cu:61-159, 886-1056), and steps k by fixed
// strides with host backups and rollbacks (src/kc.cu:1140-1309); the result
// is the same kmax and edge count.
#include <algorithm>
#include <chrono>
#include <memory>

#include "compact.cuh"
#include "dense.cuh"
#include "rows.cuh"
#include "subgraph.h"
#include "teams.h"

namespace kt {
namespace {

constexpr unsigned kPeelThreads = 256;   // host-stepped rounds
constexpr unsigned kLevelThreads = 512;  // k_levels, or fewer where the rows' shared memory wants it
constexpr unsigned kCounters = 16;   // device counters before the blocks' kept counts
constexpr unsigned kMaxGrid = 4096;  // blocks of a cooperative launch at most (one count per block is kept)

struct PeelArgs {
  const uint64_t* ends;
  const uint64_t* off;
  const uint32_t* adj;
  const uint32_t* eid;
  uint32_t n;       // vertices
  uint32_t* sup;
  uint32_t* state;
  uint32_t* truss;  // may be null
  const uint32_t* alive;
  uint64_t na;
  uint32_t* front[2];
  // [0..2] rotating frontier counters, [3..4] long rows of a list-mode round,
  // [6..7] recount cursors, [8..10] and
  // [12..14] a level's figures (k_levels, by level parity: 2^32 - 1 - the least
  // support left, the largest, the edges left), [16...] one kept count per block
  unsigned long long* cnt;
  uint64_t cap;
  uint32_t thr;    // remove support < thr
  uint32_t tval;   // trussness recorded for removed edges
  uint32_t r0;     // first round number
  uint32_t* adeg;  // alive degree per vertex (for the byte accounting)
  DenseRows R;     // dense mode: alive adjacency bitsets (R.bits null otherwise)
  float wavg;      // mean words per bitset row
  uint64_t bit0 = 0, bit_words;  // first and number of the bitset rows' words (multiples of 4)
  uint32_t gamma;  // recount round when nf * thr * gamma > alive * wavg
  uint32_t search_ratio;  // binary-search the long row when it is this many times longer
  uint32_t split;         // split rounds when frontier x chunks <= split x warps (0 = never)
  unsigned long long* acct;  // [0] sum of alive degrees of deleted edges, [1] decrements, [2] recounted edges
  DevWords* words;
  unsigned long long timeout_ns;
  // Batched unions: per-graph thresholds gthr[egr[e]] replace thr (0 = the
  // graph is finished and its edges are never frontier edges).
  const uint32_t* gthr;
  const uint32_t* egr;
  const uint32_t* gthr_max;  // batched: the largest running threshold (recount cost model)
  // List mode: the edges in a hash table (null: none), tag << 32 | edge id per
  // slot, and the frontier edges whose shorter row is long.
  const unsigned long long* table;
  uint32_t table_bits;  // 2^table_bits slots
  uint32_t* big;
  // and the rows, each of rlen[v] entries from off[v] on (with `pack`, copies
  // that k_levels may drop dead entries from).
  uint32_t* radj;
  uint32_t* reid;
  uint32_t* rlen;
  bool pack;
  // A level tried from a snapshot: give up (the level's truss is empty) as
  // soon as fewer than this many edges can remain, t(t-1)/2 for level t
  // (0: peel to the end).  The state is then partial; the caller undoes it.
  uint64_t fail_below = 0;
};

// The level in progress (k_levels changes it; the rest of PeelArgs stays).
struct Level {
  const uint32_t* alive;
  uint64_t na;
  uint32_t thr, tval;
};
__device__ __forceinline__ Level first_level(const PeelArgs& A) { return Level{A.alive, A.na, A.thr, A.tval}; }

__device__ __forceinline__ uint32_t edge_thr(const PeelArgs& A, const Level& V, uint32_t e) {
  return A.gthr ? A.gthr[A.egr[e]] : V.thr;
}

__device__ __forceinline__ void push_warp_full(bool want, uint32_t item, uint32_t* list, unsigned long long* cnt,
                                               uint64_t cap, uint32_t* err) {
  const unsigned b = __ballot_sync(kFull, want);
  if (!b) return;
  const unsigned leader = __ffs(b) - 1;
  unsigned long long base = 0;
  if (lane_id() == leader) base = atomicAdd(cnt, (unsigned long long)__popc(b));
  base = __shfl_sync(kFull, base, leader);
  if (want) {
    const unsigned long long p = base + __popc(b & lanemask_lt());
    if (p < cap)
      list[p] = item;
    else
      atomicOr(err, kDevErrCapacity);
  }
}

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

// Triangle {e, a, b} seen from frontier edge e in round r; returns which of
// a, b crossed below the threshold (to be pushed).
__device__ __forceinline__ void close_triangle(const PeelArgs& A, const Level& V, uint32_t e, uint32_t a, uint32_t b,
                                               uint32_t r, uint32_t thr, bool& pa, bool& pb, uint32_t& ndec) {
  const uint32_t sa = A.state[a], sb = A.state[b];
  if (sa < r || sb < r) return;  // broken in an earlier round
  if (sa > r && !(sb == r && b < e)) {
    ++ndec;
    if (atomicSub(&A.sup[a], 1u) == thr) {
      A.state[a] = r + 1;
      if (A.truss) A.truss[a] = V.tval;
      pa = true;
    }
  }
  if (sb > r && !(sa == r && a < e)) {
    ++ndec;
    if (atomicSub(&A.sup[b], 1u) == thr) {
      A.state[b] = r + 1;
      if (A.truss) A.truss[b] = V.tval;
      pb = true;
    }
  }
}

// Position of the r-th (from 0) set bit of m.
__device__ __forceinline__ uint32_t select_bit(uint32_t m, uint32_t r) {
  uint32_t pos = 0;
#pragma unroll
  for (uint32_t s = 16; s >= 1; s >>= 1) {
    const uint32_t low = __popc(m & ((1u << s) - 1u));
    if (r >= low) {
      r -= low;
      m >>= s;
      pos += s;
    }
  }
  return pos;
}

// Words [w0, w0 + cw) (cw at most 32) of frontier edge e's two bitset rows:
// the common neighbours found there are dealt one per lane (a warp scan of the
// words' popcounts, then a search for each task's word and a select of its
// bit), each closing its triangle.  Each common neighbour's edge ids come from
// its position in the sorted rows, a popcount of the rows as built.  Bits of
// edges deleted in earlier cascades are clear; deletions of this cascade are
// caught by close_triangle's state test.  (With each lane closing the set bits
// of its own word, a step of 32 words took as many iterations as the fullest
// word has bits: 64 mix graphs, 741 decrement rounds, 23.7 ms; dealt 15.2 ms.)
__device__ __forceinline__ void close_common(const PeelArgs& A, const Level& V, uint32_t e, uint32_t x, uint32_t y,
                                             uint32_t thr, uint32_t W, uint32_t w0, uint32_t cw, uint32_t r,
                                             uint32_t* next, unsigned long long* ncnt, uint32_t& ndec) {
  const unsigned lane = lane_id();
  const uint32_t i = w0 + lane;
  uint32_t m = 0;
  if (lane < cw && i < W) m = __ldcg(A.R.bits + A.R.off(x) + i) & __ldcg(A.R.bits + A.R.off(y) + i);
  const uint32_t c = __popc(m);
  const uint32_t incl = warp_incl_scan(c);
  const uint32_t T = __shfl_sync(kFull, incl, 31);
  if (T == 0) return;
  const uint32_t excl = incl - c;
  const uint64_t ox = A.off[x], oy = A.off[y];
  for (uint32_t base = 0; base < T; base += 32) {
    const uint32_t t = base + lane;
    uint32_t lo = 0;  // the last word whose first task is at or before t
#pragma unroll
    for (uint32_t st = 16; st >= 1; st >>= 1) {
      const uint32_t ec = __shfl_sync(kFull, excl, lo + st);
      if (ec <= t) lo += st;
    }
    const uint32_t oexcl = __shfl_sync(kFull, excl, lo), om = __shfl_sync(kFull, m, lo);
    bool pa = false, pb = false;
    uint32_t a = 0, b = 0;
    if (t < T) {
      const uint32_t col = (w0 + lo) * 32 + select_bit(om, t - oexcl);
      a = A.eid[ox + A.R.rank(x, col)];
      b = A.eid[oy + A.R.rank(y, col)];
      close_triangle(A, V, e, a, b, r, thr, pa, pb, ndec);
    }
    push_warp_full(pa, a, next, ncnt, A.cap, &A.words->err);
    push_warp_full(pb, b, next, ncnt, A.cap, &A.words->err);
  }
}

// The whole rows, each lane closing the set bits of its own words: where a
// frontier edge has far fewer common neighbours (at most thr) than its rows have
// words, a step of 32 words has few and hardly two in a word, and dealing them
// costs more than it spreads (36M edges on 60,000 vertices, thresholds up to 23,
// rows of 1,876 words: 1,530 -> 1,330 ms; 1.2M on 12,000: 4.9 -> 4.3; with a
// line at 4 instead of 8 words a neighbour the same).
constexpr uint32_t kOwnWords = 8;

__device__ __forceinline__ void close_own_words(const PeelArgs& A, const Level& V, uint32_t e, uint32_t x, uint32_t y,
                                                uint32_t thr, uint32_t W, uint32_t r, uint32_t* next,
                                                unsigned long long* ncnt, uint32_t& ndec) {
  const uint32_t *rx = A.R.bits + A.R.off(x), *ry = A.R.bits + A.R.off(y);
  const uint64_t ox = A.off[x], oy = A.off[y];
  for (uint32_t i = lane_id(); i < ((W + 31) & ~31u); i += 32) {
    uint32_t m = i < W ? __ldcg(rx + i) & __ldcg(ry + i) : 0u;
    while (__any_sync(kFull, m)) {
      bool pa = false, pb = false;
      uint32_t a = 0, b = 0;
      if (m) {
        const uint32_t col = i * 32 + __ffs(m) - 1;
        m &= m - 1;
        a = A.eid[ox + A.R.rank(x, col)];
        b = A.eid[oy + A.R.rank(y, col)];
        close_triangle(A, V, e, a, b, r, thr, pa, pb, ndec);
      }
      push_warp_full(pa, a, next, ncnt, A.cap, &A.words->err);
      push_warp_full(pb, b, next, ncnt, A.cap, &A.words->err);
    }
  }
}

// One frontier edge, one warp.  Pushes into next / ncnt; adds the edge's
// alive degrees and its decrements to the per-thread tallies.
__device__ __forceinline__ void peel_edge(const PeelArgs& A, const Level& V, uint32_t e, uint32_t r, uint32_t* next,
                                          unsigned long long* ncnt, uint64_t& tdeg, uint64_t& tdec) {
  const uint64_t k = A.ends[e];
  uint32_t x = (uint32_t)(k >> 32), y = (uint32_t)k;
  if (lane_id() == 0) tdeg += (uint64_t)atomicSub(&A.adeg[x], 1u) + atomicSub(&A.adeg[y], 1u);
  const uint32_t thr = edge_thr(A, V, e);  // the triangle's edges share e's graph
  uint32_t ndec = 0;
  uint64_t xb = A.off[x], xe = A.off[x + 1], yb = A.off[y], ye = A.off[y + 1];
  if (xe - xb > ye - yb) {
    uint64_t t = xb;
    xb = yb;
    yb = t;
    t = xe;
    xe = ye;
    ye = t;
  }
  const uint64_t na = xe - xb, nb = ye - yb;
  uint32_t* err = &A.words->err;
  const unsigned lane = lane_id();
  if (A.R.sbits && (uint64_t)A.R.words(x) <= na + nb) {
    // Dense rows shorter than the two lists: AND the two bitset rows, 32
    // words a step.
    const uint32_t W = A.R.words(x);
    if (W >= kOwnWords * thr) {
      close_own_words(A, V, e, x, y, thr, W, r, next, ncnt, ndec);
    } else {
      for (uint32_t w0 = 0; w0 < W; w0 += 32) close_common(A, V, e, x, y, thr, W, w0, 32, r, next, ncnt, ndec);
    }
    tdec += ndec;
    return;
  }
  if (nb > (uint64_t)A.search_ratio * na) {
    // Short row against a long one: binary search per lane.
    for (uint64_t q = xb + lane; q < xb + ((na + 31) & ~31ULL); q += 32) {
      bool pa = false, pb = false;
      uint32_t a = 0, b = 0;
      if (q < xe) {
        const uint64_t p = find_sorted(A.adj, yb, ye, A.adj[q]);
        if (p != ye) {
          a = A.eid[q];
          b = A.eid[p];
          close_triangle(A, V, e, a, b, r, thr, pa, pb, ndec);
        }
      }
      push_warp_full(pa, a, next, ncnt, A.cap, err);
      push_warp_full(pb, b, next, ncnt, A.cap, err);
    }
    tdec += ndec;
    return;
  }
  // Tile merge.
  uint64_t i = 0, j = 0;
  while (i < na && j < nb) {
    const uint32_t ta = (uint32_t)(na - i < 32 ? na - i : 32), tb = (uint32_t)(nb - j < 32 ? nb - j : 32);
    const uint32_t av = lane < ta ? A.adj[xb + i + lane] : 0xffffffffu;
    const uint32_t bv = lane < tb ? A.adj[yb + j + lane] : 0xffffffffu;
    const uint32_t alast = __shfl_sync(kFull, av, ta - 1);
    const uint32_t blast = __shfl_sync(kFull, bv, tb - 1);
    // Lower bound of av in the B tile (lanes < tb hold it, ascending).
    uint32_t q = 0;
#pragma unroll
    for (uint32_t s = 16; s >= 1; s >>= 1) {
      const uint32_t probe = __shfl_sync(kFull, bv, (q + s - 1) & 31);
      if (q + s <= tb && probe < av) q += s;
    }
    const uint32_t hit = __shfl_sync(kFull, bv, q & 31);
    bool pa = false, pb = false;
    uint32_t a = 0, b = 0;
    if (lane < ta && q < tb && hit == av) {
      a = A.eid[xb + i + lane];
      b = A.eid[yb + j + q];
      close_triangle(A, V, e, a, b, r, thr, pa, pb, ndec);
    }
    push_warp_full(pa, a, next, ncnt, A.cap, err);
    push_warp_full(pb, b, next, ncnt, A.cap, err);
    if (alast <= blast) i += ta;
    if (blast <= alast) j += tb;
  }
  tdec += ndec;
}

// ---- list mode: triangles of a frontier edge through an edge hash table.

__device__ __forceinline__ uint32_t edge_hash(uint32_t u, uint32_t v) {
  uint32_t h = (u * 0x9E3779B1u) ^ __funnelshift_l(v * 0x85EBCA77u, v * 0x85EBCA77u, 15);
  h ^= h >> 15;
  return h * 0xC2B2AE3Du;
}
__device__ __forceinline__ uint32_t edge_tag(uint32_t u, uint32_t v) { return (u * 0x27D4EB2Fu) ^ (v + (v << 13)); }
constexpr unsigned long long kNoEdge = ~0ULL;

__global__ void k_row_lengths(const uint64_t* __restrict__ off, uint64_t n, uint32_t* __restrict__ len) {
  for (uint64_t v = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; v < n; v += (uint64_t)gridDim.x * blockDim.x)
    len[v] = (uint32_t)(off[v + 1] - off[v]);
}

__global__ void k_table_build(uint64_t m, const uint64_t* __restrict__ ends, unsigned long long* table,
                              uint32_t bits) {
  const uint64_t mask = (1ULL << bits) - 1;
  for (uint64_t e = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; e < m; e += (uint64_t)gridDim.x * blockDim.x) {
    const uint64_t k = ends[e];
    const uint32_t u = (uint32_t)(k >> 32), v = (uint32_t)k;
    const unsigned long long ent = ((unsigned long long)edge_tag(u, v) << 32) | (uint32_t)e;
    uint64_t at = edge_hash(u, v) >> (32 - bits);
    while (atomicCAS(&table[at], kNoEdge, ent) != kNoEdge) at = (at + 1) & mask;  // at most 2/5 of the slots fill
  }
}

// Id of the edge (a, b), or 0xffffffff.
__device__ __forceinline__ uint32_t find_edge(const PeelArgs& A, uint32_t a, uint32_t b) {
  const uint32_t u = min(a, b), v = max(a, b), tag = edge_tag(u, v);
  const uint64_t key = ((uint64_t)u << 32) | v, mask = (1ULL << A.table_bits) - 1;
  for (uint64_t at = edge_hash(u, v) >> (32 - A.table_bits);; at = (at + 1) & mask) {
    const unsigned long long ent = A.table[at];
    if (ent == kNoEdge) return 0xffffffffu;
    if ((uint32_t)(ent >> 32) == tag && A.ends[(uint32_t)ent] == key) return (uint32_t)ent;
  }
}

// The end of edge (x, y) with the shorter row.
__device__ __forceinline__ void shorter_row(const PeelArgs& A, uint32_t e, uint32_t& s, uint32_t& other) {
  const uint64_t k = A.ends[e];
  s = (uint32_t)(k >> 32);
  other = (uint32_t)k;
  if (A.rlen[s] > A.rlen[other]) {
    const uint32_t t = s;
    s = other;
    other = t;
  }
}

// N row entries per lane (row positions j[t], where ok[t]) of the shorter rows
// of frontier edges e[t], whose other ends are o[t].  (Looking the third edges
// up before the entries' own states are known, an access less in a small
// round's chain, costs more for the dead entries than it saves.)
template <unsigned N>
__device__ __forceinline__ void close_entries(const PeelArgs& A, const Level& V, const uint32_t (&e)[N],
                                              const uint32_t (&o)[N], const uint64_t (&j)[N], const bool (&ok)[N],
                                              uint32_t r, uint32_t* next, unsigned long long* ncnt, uint32_t& ndec) {
  uint32_t a[N], w[N], b[N];
#pragma unroll
  for (unsigned t = 0; t < N; ++t) {
    a[t] = ok[t] ? A.reid[j[t]] : 0u;
    w[t] = ok[t] ? A.radj[j[t]] : 0u;
  }
  bool live[N];
#pragma unroll
  for (unsigned t = 0; t < N; ++t) live[t] = ok[t] && a[t] != e[t] && A.state[a[t]] >= r;
#pragma unroll
  for (unsigned t = 0; t < N; ++t) b[t] = live[t] ? find_edge(A, o[t], w[t]) : 0xffffffffu;
#pragma unroll
  for (unsigned t = 0; t < N; ++t) {
    bool pa = false, pb = false;
    if (b[t] != 0xffffffffu) close_triangle(A, V, e[t], a[t], b[t], r, edge_thr(A, V, e[t]), pa, pb, ndec);
    __syncwarp();
    push_warp_full(pa, a[t], next, ncnt, A.cap, &A.words->err);
    push_warp_full(pb, b[t], next, ncnt, A.cap, &A.words->err);
  }
}

// Drops the dead entries of every row, in place, a warp per row.
__device__ __forceinline__ void pack_rows(const PeelArgs& A, uint64_t gwarp, uint64_t gwarps) {
  const unsigned lane = lane_id();
  for (uint64_t v = gwarp; v < A.n; v += gwarps) {
    const uint64_t b = A.off[v];
    const uint32_t len = A.rlen[v];
    uint32_t kept = 0;
    for (uint32_t j0 = 0; j0 < len; j0 += 32) {
      const uint32_t j = j0 + lane;
      const uint32_t e = j < len ? A.reid[b + j] : 0u, w = j < len ? A.radj[b + j] : 0u;
      const bool keep = j < len && A.state[e] == kAlive;
      const unsigned bal = __ballot_sync(kFull, keep);
      __syncwarp();
      if (keep) {
        const uint64_t at = b + kept + __popc(bal & lanemask_lt());
        A.reid[at] = e;
        A.radj[at] = w;
      }
      kept += __popc(bal);
    }
    if (lane == 0) A.rlen[v] = kept;
  }
}

// A round over the frontier's shorter rows.  A frontier of at most kBigBatch
// edges has the windows of all its rows dealt to every warp at once: every block
// adds up the rows' lengths by itself, which is one batch of deal_windows, and
// no warp is left with a row of many steps.  Of a larger one, a warp takes up to
// 32 edges and walks their rows end to end; rows of more than kLongJob entries
// go to A.big[0..*nbig), whose windows are dealt after a barrier.  An entry
// costs its edge's state and, if that is alive, one table slot or two, all
// independent of its neighbours'; the merge of the two sorted rows by one warp
// was a chain of as many dependent steps as the rows have tiles of 32 entries
// (truss numbers of an R-MAT scale 16 graph, 850,000 edges, 828 rounds: levels
// 52.2 -> 15.9 ms, with small frontiers dealt 12.4, now 11.0; dealing up to
// 4,096 edges so is slower by 0.4).
constexpr uint32_t kLongJob = 256;
constexpr unsigned kJobWide = 2;

__device__ __forceinline__ void list_round(const PeelArgs& A, const Level& V, const uint32_t* fr, uint64_t nf,
                                           uint32_t r, uint32_t* next, unsigned long long* ncnt,
                                           unsigned long long* nbig, uint64_t& tdeg, uint64_t& tdec) {
  const uint64_t gwarps = (uint64_t)gridDim.x * (blockDim.x >> 5);
  const uint64_t gwarp = (uint64_t)blockIdx.x * (blockDim.x >> 5) + warp_id();
  const unsigned lane = lane_id();
  const uint64_t share = (nf + gwarps - 1) / gwarps;
  const uint32_t per = share < 32 ? (uint32_t)share : 32u;
  uint32_t ndec = 0;
  for (uint64_t f0 = gwarp * per; f0 < nf; f0 += gwarps * per) {
    uint64_t start = 0;
    uint32_t len = 0, e = 0, o = 0;
    bool is_long = false;
    if (lane < per && f0 + lane < nf) {
      e = fr[f0 + lane];
      uint32_t s;
      shorter_row(A, e, s, o);
      tdeg += (uint64_t)atomicSub(&A.adeg[s], 1u) + atomicSub(&A.adeg[o], 1u);
      start = A.off[s];
      const uint32_t l = A.rlen[s];
      is_long = l > kLongJob;
      len = is_long ? 0u : l;
    }
    push_warp_full(is_long, e, A.big, nbig, A.cap, &A.words->err);
    const uint32_t incl = warp_incl_scan(len);
    const uint32_t total = __shfl_sync(kFull, incl, 31), excl = incl - len;
    start -= excl;  // entry p of the walk is at start + p of its row's lane
    for (uint32_t base = 0; base < total; base += 32 * kJobWide) {
      uint32_t ee[kJobWide], oo[kJobWide];
      uint64_t j[kJobWide];
      bool ok[kJobWide];
#pragma unroll
      for (unsigned t = 0; t < kJobWide; ++t) {
        const uint32_t p = base + 32 * t + lane;
        uint32_t from = 0;  // the last row starting at or before p
        if (per > 1) {
#pragma unroll
          for (uint32_t st = 16; st >= 1; st >>= 1) {
            const uint32_t x = __shfl_sync(kFull, excl, from + st);
            if (x <= p) from += st;
          }
        }
        ee[t] = __shfl_sync(kFull, e, from);
        oo[t] = __shfl_sync(kFull, o, from);
        j[t] = __shfl_sync(kFull, start, from) + p;
        ok[t] = p < total;
      }
      close_entries<kJobWide>(A, V, ee, oo, j, ok, r, next, ncnt, ndec);
    }
  }
  tdec += ndec;
}

// The shorter rows of up to kBigBatch frontier edges, in shared memory: each
// edge and its other end, where the row starts, how long it is, and the first of
// its windows.
struct RowBatch {
  uint64_t start[kBigBatch];
  uint32_t first[kBigBatch + 1], len[kBigBatch], edge[kBigBatch], other[kBigBatch];
  uint32_t tmp[33];
};

// The windows of the shorter rows of edges[0..n), dealt to every warp.  As
// deal_windows, but a warp finds its window's row in shared memory: from the
// frontier through the edges to the offsets is a chain of three accesses, which
// every window would go through again (828 rounds: 12.4 -> 12.1 ms).
__device__ __forceinline__ void list_round_windows(const PeelArgs& A, const Level& V, const uint32_t* edges,
                                                   uint64_t n, uint32_t r, uint32_t* next, unsigned long long* ncnt,
                                                   RowBatch& B, uint64_t& tdec) {
  constexpr uint32_t kWin = 32 * kJobWide;
  const uint32_t gwarps = gridDim.x * (blockDim.x >> 5), gwarp = blockIdx.x * (blockDim.x >> 5) + warp_id();
  const uint32_t per = kBigBatch / blockDim.x;  // rows per thread
  uint32_t ndec = 0;
  for (uint64_t base = 0; base < n; base += kBigBatch) {
    const uint32_t cnt = (uint32_t)min((uint64_t)kBigBatch, n - base);
    uint32_t sum = 0;
    for (uint32_t j = 0; j < per; ++j) {
      const uint32_t x = threadIdx.x * per + j;
      if (x >= cnt) break;
      const uint32_t e = edges[base + x];
      uint32_t s, o;
      shorter_row(A, e, s, o);
      const uint32_t l = A.rlen[s];
      B.start[x] = A.off[s];
      B.len[x] = l;
      B.edge[x] = e;
      B.other[x] = o;
      sum += (l + kWin - 1) / kWin;
    }
    uint32_t total;
    uint32_t pre = block_excl_scan<uint32_t>(sum, B.tmp, &total);
    for (uint32_t j = 0; j < per; ++j) {
      const uint32_t x = threadIdx.x * per + j;
      if (x >= cnt) break;
      B.first[x] = pre;
      pre += (B.len[x] + kWin - 1) / kWin;
    }
    __syncthreads();
    for (uint32_t u = gwarp; u < total; u += gwarps) {
      uint32_t lo = 0, hi = cnt;  // last row with first <= u
      while (hi - lo > 1) {
        const uint32_t mid = (lo + hi) >> 1;
        if (B.first[mid] <= u)
          lo = mid;
        else
          hi = mid;
      }
      const uint32_t at = (u - B.first[lo]) * kWin, len = B.len[lo];
      uint32_t ee[kJobWide], oo[kJobWide];
      uint64_t j[kJobWide];
      bool ok[kJobWide];
#pragma unroll
      for (unsigned t = 0; t < kJobWide; ++t) {
        const uint32_t p = at + 32 * t + lane_id();
        ee[t] = B.edge[lo];
        oo[t] = B.other[lo];
        j[t] = B.start[lo] + p;
        ok[t] = p < len;
      }
      close_entries<kJobWide>(A, V, ee, oo, j, ok, r, next, ncnt, ndec);
    }
    __syncthreads();
  }
  tdec += ndec;
}

// A decrement round over (frontier edge, chunk of cw words) units, a warp
// each, so a small frontier of edges with many triangles keeps the whole grid
// busy (a round of one edge in a core of 1,311 vertices: 13.2 us in chunks of 8
// words, 5.4 us in the shortest that fill the grid); edges that use the
// sorted-list merge go whole to the warp of their first chunk.
constexpr uint32_t kSplitWords = 8;  // words of a chunk at most

__device__ __forceinline__ void split_round(const PeelArgs& A, const Level& V, const uint32_t* fr, uint32_t nf,
                                            uint32_t cw, uint32_t chunks, uint32_t r, uint32_t* next,
                                            unsigned long long* ncnt, uint32_t gwarp, uint32_t gwarps,
                                            uint64_t& tdeg, uint64_t& tdec) {
  uint32_t ndec = 0;
  for (uint32_t u = gwarp; u < nf * chunks; u += gwarps) {
    const uint32_t f = u / chunks;
    const uint32_t ch = u - f * chunks;
    const uint32_t e = fr[f];
    const uint64_t k = A.ends[e];
    const uint32_t x = (uint32_t)(k >> 32), y = (uint32_t)k;
    const uint64_t na = A.off[x + 1] - A.off[x], nb = A.off[y + 1] - A.off[y];
    const uint32_t W = A.R.words(x);
    if ((uint64_t)W > na + nb) {  // peel_edge would merge the lists
      if (ch == 0) peel_edge(A, V, e, r, next, ncnt, tdeg, tdec);
      continue;
    }
    if (ch * cw >= W) continue;
    if (ch == 0 && lane_id() == 0) tdeg += (uint64_t)atomicSub(&A.adeg[x], 1u) + atomicSub(&A.adeg[y], 1u);
    close_common(A, V, e, x, y, edge_thr(A, V, e), W, ch * cw, cw, r, next, ncnt, ndec);
  }
  tdec += ndec;
}

__device__ __forceinline__ void flush_tallies(const PeelArgs& A, uint64_t tdeg, uint64_t tdec) {
  tdeg = warp_sum(tdeg);
  tdec = warp_sum(tdec);
  if (lane_id() == 0) {
    if (tdeg) atomicAdd(&A.acct[0], (unsigned long long)tdeg);
    if (tdec) atomicAdd(&A.acct[1], (unsigned long long)tdec);
  }
}

// Frontier of a level: alive edges with support below the threshold.  (Four
// entries per thread in flight: the passes over the alive list wait for three
// dependent loads each, and are most of a level that removes a few edges.)
constexpr unsigned kListWide = 4;

__device__ __forceinline__ void level_frontier(const PeelArgs& A, const Level& V, uint32_t r, uint32_t* front,
                                               unsigned long long* cnt, uint64_t gtid, uint64_t gthreads) {
  for (uint64_t i0 = gtid & ~31ULL; i0 < V.na; i0 += kListWide * gthreads) {
    uint32_t e[kListWide];
    bool want[kListWide];
#pragma unroll
    for (unsigned t = 0; t < kListWide; ++t) {
      const uint64_t i = i0 + t * gthreads + lane_id();
      want[t] = i < V.na;
      e[t] = want[t] ? V.alive[i] : 0u;
    }
#pragma unroll
    for (unsigned t = 0; t < kListWide; ++t)
      want[t] = want[t] && A.state[e[t]] == kAlive && A.sup[e[t]] < edge_thr(A, V, e[t]);
#pragma unroll
    for (unsigned t = 0; t < kListWide; ++t) {
      if (want[t]) {
        A.state[e[t]] = r;
        if (A.truss) A.truss[e[t]] = V.tval;
      }
      push_warp_full(want[t], e[t], front, cnt, A.cap, &A.words->err);
    }
  }
}

__device__ __forceinline__ void clear_edge_bits(const PeelArgs& A, uint32_t e) {
  const uint64_t k = A.ends[e];
  const uint32_t x = (uint32_t)(k >> 32), y = (uint32_t)k;
  const uint32_t cy = A.R.col(x, y), cx = A.R.col(y, x);
  atomicAnd(&A.R.bits[A.R.off(x) + (cy >> 5)], ~(1u << (cy & 31)));
  atomicAnd(&A.R.bits[A.R.off(y) + (cx >> 5)], ~(1u << (cx & 31)));
}

// Rebuilds the bitsets from the surviving edges when more edges were deleted
// since the bits were last current than survive: zero every word, then (after
// a grid barrier, in the caller) set the bits of the alive-list edges still
// alive -- fewer atomics than clearing the deleted edges one by one.
__device__ __forceinline__ void zero_bits(const PeelArgs& A, uint64_t gtid, uint64_t gthreads) {
  uint4* p = reinterpret_cast<uint4*>(A.R.bits + A.bit0);
  for (uint64_t w = gtid; w < A.bit_words / 4; w += gthreads) p[w] = make_uint4(0u, 0u, 0u, 0u);
}
__device__ __forceinline__ void set_alive_bits(const PeelArgs& A, const Level& V, uint64_t gtid, uint64_t gthreads) {
  for (uint64_t i = gtid; i < V.na; i += gthreads) {
    const uint32_t e = V.alive[i];
    if (A.state[e] != kAlive) continue;
    const uint64_t k = A.ends[e];
    const uint32_t x = (uint32_t)(k >> 32), y = (uint32_t)k;
    const uint32_t cy = A.R.col(x, y), cx = A.R.col(y, x);
    atomicOr(&A.R.bits[A.R.off(x) + (cy >> 5)], 1u << (cy & 31));
    atomicOr(&A.R.bits[A.R.off(y) + (cx >> 5)], 1u << (cx & 31));
  }
}

// Clears the bits of alive-list edges deleted in rounds (lo, hi].
__device__ __forceinline__ void clear_deleted(const PeelArgs& A, const Level& V, uint32_t lo, uint32_t hi, uint64_t gtid,
                                              uint64_t gthreads) {
  for (uint64_t i = gtid; i < V.na; i += gthreads) {
    const uint32_t e = V.alive[i];
    const uint32_t st = A.state[e];
    if (st > lo && st <= hi) clear_edge_bits(A, e);
  }
}

// Shared memory of a k_levels block's rows at most (its static arrays and the
// block's reserve take some of the 227 KB).
constexpr size_t kRowsSmem = 200 << 10;

constexpr uint64_t kRowsInL2 = 64u << 20;  // bytes of bitset rows that stay in L2 beside the rest

// Dense recount round r: every surviving edge gets its exact support in the
// graph without this round's frontier; those below the threshold form the
// next frontier.  Replaces per-triangle decrements when the frontier is a
// large part of the graph.
// A group is 32 entries of the alive list, or fewer (8 at least) where that
// leaves warps of the grid without one: its edges are counted one after
// another.  Rows that fit in L2 together are read in any order, so warps
// stride over the groups; of more rows, warps take the next group from
// `cursor` (zero at the start of the round), so that the groups in flight stay
// a narrow window of the tile-ordered list -- the cursor is one word that every
// group waits for, 10 us of a 25 us round of 230,000 edges.
__device__ __forceinline__ void recount_round(const PeelArgs& A, const Level& V, uint32_t r, uint32_t* next,
                                              unsigned long long* ncnt, unsigned long long* cursor,
                                              uint64_t& trec, uint32_t* su, const Crew& crew) {
  const uint64_t gwarps = (uint64_t)crew.blocks * (blockDim.x >> 5);
  const uint64_t share = V.na / gwarps;
  const uint32_t size = share >= 128 ? 32u : share >= 64 ? 16u : 8u;
  const uint64_t groups = (V.na + size - 1) / size;
  const bool in_l2 = A.bit_words <= kRowsInL2 / 4;
  uint64_t mine = (uint64_t)crew.rank * (blockDim.x >> 5) + warp_id();
  for (;;) {
    unsigned long long g = mine;
    if (in_l2) {
      mine += gwarps;
    } else {
      if (lane_id() == 0) g = atomicAdd(cursor, 1ULL);
      g = __shfl_sync(kFull, g, 0);
    }
    if (g >= groups) break;
    uint32_t e, sc;
    bool ok;
    const uint64_t last = min(V.na, (uint64_t)(g + 1) * size);
    if (A.R.W <= kShortRow)
      dense_group_short(V.alive, g * size, last, A.ends, A.R, A.state, size / 4, e, sc, ok);
    else
      dense_group<2>(V.alive, g * size, last, A.ends, A.R, A.state, su, e, sc, ok);
    trec += __popc(__ballot_sync(kFull, ok));
    bool want = false;
    if (ok) {
      A.sup[e] = sc;
      if (sc < edge_thr(A, V, e)) {
        A.state[e] = r + 1;
        if (A.truss) A.truss[e] = V.tval;
        want = true;
      }
    }
    push_warp_full(want, e, next, ncnt, A.cap, &A.words->err);
  }
}

// What k_levels leaves for the host.
enum LevelsEnd : uint32_t {
  kEndEmpty = 0,    // no edge is left (or the level tried gave up)
  kEndLevels = 1,   // max_levels done
  kEndStop = 2,     // the first level kept exactly stop_count edges
  kEndCompact = 3,  // few enough edges are left for a smaller graph
};
struct LevelsOut {
  uint64_t na, rounds, count, scanned;
  uint32_t list;         // alive list in use (0 or 1)
  uint32_t levels;       // levels run
  uint32_t kept;         // levels that left edges
  uint32_t kmax, mn, mx; // after the last of those: its level, least and largest support
  uint32_t recounts, r_next, end, gave_up;
};

struct LevelsArgs {
  uint32_t* alive[2];       // the list in use, and the one the next is written to
  uint32_t max_levels;      // 0: until a reason to end
  uint64_t stop_count;      // end after the first level if it keeps exactly this many edges (0: no)
  uint64_t compact_at;      // end once this many edges or fewer are left (0: no)
  LevelsOut* out;
  // Batched unions (ngroups > 0): every graph's alive edges and least support
  // of a level, its record and its next threshold.
  uint32_t ngroups;
  uint32_t group0, group1;  // the graphs whose levels are recorded here
  unsigned long long* gcnt;
  uint32_t* gmin;
  uint32_t* kmax;
  uint64_t* count;
  uint32_t* gthr;
  uint32_t* tmax;
  const uint64_t* stop;
  // Teams of blocks, each with a stretch of the graphs (dense unions): the alive
  // list is in the teams' order.
  const struct PeelTeam* teams;
  uint32_t nteams;
  uint32_t counters;  // a team's words of PeelArgs::cnt
  DevWords* team_words;
};

struct PeelTeam {
  uint32_t block0, blocks;
  uint32_t group0, group1;
  uint64_t list0, na;        // its edges in the alive list
  uint64_t bit0, bit_words;  // its bitset rows
  float wavg;
};
// Rows from this many words on (16,000 vertices): blocks of 256 threads, five to
// an SM where the rows' shared memory allows, with fewer registers a thread.  Rounds
// there are mostly merges and intersections of long rows, a chain of accesses per
// warp, and take as long as there are few warps: 5M edges on 20,000 vertices 37.5 ms
// with 32 warps on an SM, 33.0 with 40; 10M on 40,000 133.9 and 122.6.  Shorter rows
// are recounted more, which spilled registers slow down.
constexpr uint32_t kWideRow = 512;
constexpr unsigned kMaxPeelTeams = 32;  // (their results are read through the context's pinned words)

__device__ __forceinline__ void record_group(uint32_t g, unsigned long long* gcnt, uint32_t* gmin, uint32_t* kmax,
                                             uint64_t* count, uint32_t* gthr, const uint64_t* stop, bool first) {
  const unsigned long long n = __ldcg(&gcnt[g]);
  const uint32_t mn = __ldcg(&gmin[g]);
  if (gthr[g]) {
    if (n) {
      kmax[g] = mn + 2;
      count[g] = n;
      gthr[g] = first && stop && stop[g] && n == stop[g] ? 0u : mn + 1;
    } else {
      gthr[g] = 0;
    }
  }
  gcnt[g] = 0;
  gmin[g] = 0xffffffffu;
}

// Truss levels in one cooperative launch, from level A.thr + 2 up: a cascade
// (frontier, then rounds), an ordered compaction of the alive list (each block
// counts and writes its own stretch of it) that also finds the least support
// left, and the next level from that.  With a launch per cascade and the
// compaction, the minimum and three host reads between two, a level that
// removes a few edges took 105 us (a core of 1,311 vertices, 609,432 edges), now
// 43 us.  Dense mode uses W words of shared memory per warp for the recount
// rounds.
// Two blocks of 512 threads per SM (of long rows: kWideRow): a barrier of 296 blocks takes 1.6 us, of 592
// blocks of 256 threads 2.3 (64 mix graphs: 29.6 -> 29.1 ms of levels; one
// block of 1024 threads waits longer for its own warps on small graphs).
//
// kTeams: the graphs of a union by teams of blocks, as in the core
// decomposition (Peeler::init_teams): 64 cores of up to 1,340 vertices, 3.9M
// edges, in step 516 rounds and 15.1 ms, by teams 232 at most and 10.7.
template <bool kLists, bool kTeams, unsigned kThreads, unsigned kBlocks>
__global__ void __launch_bounds__(kThreads, kBlocks)
    k_levels(const __grid_constant__ PeelArgs all, const __grid_constant__ LevelsArgs all_levels) {
  extern __shared__ __align__(16) uint32_t dense_smem[];
  __shared__ __align__(16) unsigned char args_store[sizeof(PeelArgs)], levels_store[sizeof(LevelsArgs)];
  __shared__ unsigned team_block0, team_blocks;
  PeelArgs& my_args = *reinterpret_cast<PeelArgs*>(args_store);
  LevelsArgs& my_levels = *reinterpret_cast<LevelsArgs*>(levels_store);
  if (kTeams) {
    if (threadIdx.x == 0) {
      uint32_t t = 0;
      while (t + 1 < all_levels.nteams && all_levels.teams[t + 1].block0 <= blockIdx.x) ++t;
      const PeelTeam T = all_levels.teams[t];
      team_block0 = T.block0;
      team_blocks = T.blocks;
      my_args = all;
      my_levels = all_levels;
      my_args.alive += T.list0;
      my_args.na = T.na;
      my_args.cap = T.na;
      my_args.front[0] += T.list0;
      my_args.front[1] += T.list0;
      my_args.cnt += (uint64_t)t * all_levels.counters;
      my_args.words = all_levels.team_words + t;
      my_args.bit0 = T.bit0;
      my_args.bit_words = T.bit_words;
      my_args.wavg = T.wavg;
      my_args.gthr_max = all.gthr_max + t;
      my_levels.alive[0] += T.list0;
      my_levels.alive[1] += T.list0;
      my_levels.group0 = T.group0;
      my_levels.group1 = T.group1;
      my_levels.tmax += t;
      my_levels.out += t;
    }
    __syncthreads();
  }
  const PeelArgs& A = kTeams ? my_args : all;
  const LevelsArgs& L = kTeams ? my_levels : all_levels;
  const Crew crew = kTeams ? Crew(blockIdx.x - team_block0, team_blocks) : Crew();
  __shared__ unsigned long long sh[3];
  __shared__ uint64_t wtmp[33];
  RowBatch* batch = reinterpret_cast<RowBatch*>(dense_smem);  // lists
  uint32_t* su = dense_smem + warp_id() * (kLists ? 0 : A.R.W);  // bitsets
  const unsigned long long* src[3] = {nullptr, nullptr, nullptr};
  const uint64_t gthreads = (uint64_t)crew.blocks * blockDim.x;
  const uint64_t gtid = (uint64_t)crew.rank * blockDim.x + threadIdx.x;
  const uint64_t gwarps = gthreads >> 5, gwarp = gtid >> 5;
  unsigned long long* kept = A.cnt + kCounters;
  Level V = first_level(A);
  uint64_t tdeg = 0, tdec = 0, trec = 0, scanned = 0, rounds = 0, rec_count = 0;
  uint32_t cleared = A.r0;  // bits are current for deletions up to this round
  uint32_t i = 0, nrec = 0, list = 0, levels = 0, nkept = 0, rec_kmax = 0, rec_mn = 0, rec_mx = 0;
  uint32_t end = kEndEmpty;
  bool gave_up = false;
  uint64_t left = V.na;  // edges alive (the list may hold dead ones too)
  uint64_t packed = V.na;  // edges alive when the rows were last packed
  while (true) {
    // Slot (i + 1) % 3 is zero; slot (i + 2) % 3, and the long rows' count
    // that the next round uses, were read before the barrier of the last round.
    if (gtid == 0) {
      A.cnt[(i + 2) % 3] = 0;
      A.cnt[3 + ((i + 1) & 1)] = 0;
    }
    scanned += V.na;
    const uint64_t before = left;
    level_frontier(A, V, A.r0 + i + 1, (i & 1) ? A.front[0] : A.front[1], &A.cnt[(i + 1) % 3], gtid, gthreads);
    ++i;
    src[0] = &A.cnt[i % 3];
    src[1] = src[2] = nullptr;
    if (!grid_barrier_read(A.words, A.timeout_ns, src, sh, crew)) return;
    // The next level's figures, last read before this barrier.
    unsigned long long* fig = A.cnt + 8 + 4 * (levels & 1);
    if (gtid == 0)
      for (int q = 0; q < 3; ++q) A.cnt[8 + 4 * ((levels + 1) & 1) + q] = 0;
    uint64_t alive = before;
    uint64_t pending = 0;  // edges deleted since the bits were current
    while (true) {
      const uint64_t nf = sh[0];
      if (nf == 0) break;
      // Every block reads the same counts, so all of them give up together.
      if (alive - nf < A.fail_below) {
        gave_up = true;
        break;
      }
      const uint32_t r = A.r0 + i;
      uint32_t* fr = (i & 1) ? A.front[1] : A.front[0];
      uint32_t* nx = (i & 1) ? A.front[0] : A.front[1];
      unsigned long long* nc = &A.cnt[(i + 1) % 3];
      if (kLists) {
        unsigned long long* bc = &A.cnt[3 + (i & 1)];
        if (nf <= kBigBatch) {
          for (uint64_t f = gtid; f < nf; f += gthreads) {
            const uint64_t k = A.ends[fr[f]];
            tdeg += (uint64_t)atomicSub(&A.adeg[(uint32_t)(k >> 32)], 1u) + atomicSub(&A.adeg[(uint32_t)k], 1u);
          }
          list_round_windows(A, V, fr, nf, r, nx, nc, *batch, tdec);
        } else {
          list_round(A, V, fr, nf, r, nx, nc, bc, tdeg, tdec);
        }
        if (gtid == 0) {
          A.cnt[(i + 2) % 3] = 0;        // read at the start of round i-1
          A.cnt[3 + ((i + 1) & 1)] = 0;  // long rows of round i-1, read before the barrier ending it
        }
        src[0] = nc;
        src[1] = bc;
        if (!grid_barrier_read(A.words, A.timeout_ns, src, sh, crew)) return;
        const uint64_t nbig = sh[1];
        if (nbig) {
          list_round_windows(A, V, A.big, nbig, r, nx, nc, *batch, tdec);
          if (!grid_barrier_read(A.words, A.timeout_ns, src, sh, crew)) return;
        }
        alive -= nf;
        ++i;
        ++rounds;
        continue;
      }
      const uint32_t thr = A.gthr_max ? __ldcg(A.gthr_max) : V.thr;
      // (A factor of 2 for unions with rows beyond the short ones, whose graphs'
      // thresholds are at most thr, many of them well below it: 64 mix graphs in a
      // batch 167.9 ms without it, 163.9 with 2, 165.4 with 5.  For one graph thr is
      // its own: 8.5M edges on 12,000 vertices 43 ms without a factor, 58 with 2; the
      // Chung-Lu solve, short rows, 18.0 and 18.2.)
      const double scale = A.gthr && A.R.W > kShortRow ? 2.0 : 1.0;
      const bool recount = A.R.bits && (double)nf * (double)(thr > 0 ? thr : 1) * (double)A.gamma >
                                           scale * (double)alive * (double)A.wavg;
      pending += nf;
      if (recount) {
        ++nrec;
        // Group cursors: this recount uses slot 6 + (nrec & 1); the other slot,
        // last used by the previous recount (finished before the barrier that
        // ended its round), is cleared for the next one.
        if (gtid == 0) A.cnt[6 + ((nrec + 1) & 1)] = 0;
        if (pending > alive - nf) {
          zero_bits(A, gtid, gthreads);
          if (!grid_barrier(A.words, A.timeout_ns, crew)) return;
          set_alive_bits(A, V, gtid, gthreads);
        } else if (cleared + 1 == r) {  // only this round's frontier to clear
          for (uint64_t f = gtid; f < nf; f += gthreads) clear_edge_bits(A, fr[f]);
        } else {
          clear_deleted(A, V, cleared, r, gtid, gthreads);
        }
        cleared = r;
        pending = 0;
        if (!grid_barrier(A.words, A.timeout_ns, crew)) return;
        recount_round(A, V, r, nx, nc, &A.cnt[6 + (nrec & 1)], trec, su, crew);
      } else {
        // Few frontier edges for the grid: deal (edge, chunk) units instead,
        // in the shortest chunks that give every warp one unit at most (a
        // chunk's common neighbours, up to 32 a word, are closed 32 at a time).
        const uint64_t chunks = A.R.sbits ? (A.R.W + kSplitWords - 1) / kSplitWords : 1;
        if (A.R.sbits && A.R.W >= 2 && nf * chunks <= (uint64_t)A.split * gwarps) {
          uint32_t cw = 1;
          while (cw < kSplitWords && nf * ((A.R.W + cw - 1) / cw) > gwarps) cw *= 2;
          split_round(A, V, fr, (uint32_t)nf, cw, (A.R.W + cw - 1) / cw, r, nx, nc, (uint32_t)gwarp,
                      (uint32_t)gwarps, tdeg, tdec);
        } else
          for (uint64_t f = gwarp; f < nf; f += gwarps) peel_edge(A, V, fr[f], r, nx, nc, tdeg, tdec);
      }
      if (gtid == 0) A.cnt[(i + 2) % 3] = 0;  // read at the start of round i-1, next written in round i+1
      src[0] = nc;
      if (!grid_barrier_read(A.words, A.timeout_ns, src, sh, crew)) return;
      alive -= nf;
      ++i;
      ++rounds;
    }
    ++levels;
    if (gave_up || alive == 0) break;
    // Bring the bitsets up to date with this cascade's remaining deletions.
    if (!kLists && A.R.bits && pending) {
      if (pending > alive) {
        zero_bits(A, gtid, gthreads);
        if (!grid_barrier(A.words, A.timeout_ns, crew)) return;
        set_alive_bits(A, V, gtid, gthreads);
      } else {
        clear_deleted(A, V, cleared, A.r0 + i, gtid, gthreads);
      }
    }
    cleared = A.r0 + i;
    // What is left, and its least and largest support.  Block b owns
    // [b, b + 1) * stretch of the list.
    const uint64_t stretch = (V.na + crew.blocks - 1) / crew.blocks;
    const uint64_t s0 = min(V.na, crew.rank * stretch), s1 = min(V.na, s0 + stretch);
    uint64_t n = 0;
    uint32_t mn = 0xffffffffu, mx = 0;
    for (uint64_t j0 = s0; j0 < s1; j0 += kListWide * blockDim.x) {
      uint32_t e[kListWide], g[kListWide], sv[kListWide];
      bool keep[kListWide];
#pragma unroll
      for (unsigned t = 0; t < kListWide; ++t) {
        const uint64_t j = j0 + t * blockDim.x + threadIdx.x;
        keep[t] = j < s1;
        e[t] = keep[t] ? V.alive[j] : 0u;
      }
#pragma unroll
      for (unsigned t = 0; t < kListWide; ++t) {
        keep[t] = keep[t] && A.state[e[t]] == kAlive;
        g[t] = keep[t] && L.ngroups ? A.egr[e[t]] : 0xffffffffu;
        sv[t] = keep[t] ? A.sup[e[t]] : 0xffffffffu;
      }
#pragma unroll
      for (unsigned t = 0; t < kListWide; ++t) {
        if (L.ngroups) {
          keep[t] = keep[t] && A.gthr[g[t]] != 0;  // the edges of finished graphs do not count
          // Graphs are contiguous in the edge order: aggregate equal graphs.
          const uint32_t gr = keep[t] ? g[t] : 0xffffffffu;
          const unsigned peers = __match_any_sync(kFull, gr);
          const uint32_t gm = __reduce_min_sync(peers, keep[t] ? sv[t] : 0xffffffffu);
          if (keep[t] && lane_id() == (unsigned)(__ffs(peers) - 1)) {
            atomicAdd(&L.gcnt[gr], (unsigned long long)__popc(peers));
            atomicMin(&L.gmin[gr], gm);
          }
        }
        if (keep[t]) {
          ++n;
          mn = min(mn, sv[t]);
          mx = max(mx, sv[t]);
        }
      }
    }
    n = block_sum<uint64_t>(n, wtmp);
    mn = warp_min(mn);
    mx = warp_max(mx);
    if (lane_id() == 0 && mn != 0xffffffffu) {
      atomicMax(&fig[0], (unsigned long long)(0xffffffffu - mn));
      atomicMax(&fig[1], (unsigned long long)mx);
    }
    if (threadIdx.x == 0) {
      kept[crew.rank] = n;
      if (n) atomicAdd(&fig[2], (unsigned long long)n);
    }
    src[0] = &fig[0];
    src[1] = &fig[1];
    src[2] = &fig[2];
    if (!grid_barrier_read(A.words, A.timeout_ns, src, sh, crew)) return;
    rec_mn = 0xffffffffu - (uint32_t)sh[0];
    rec_mx = (uint32_t)sh[1];
    left = sh[2];
    ++nkept;
    rec_kmax = rec_mn + 2;
    rec_count = left;
    if (L.ngroups) {
      if (left == 0) {
        end = kEndEmpty;
        break;
      }
    } else {
      if (L.stop_count && nkept == 1 && left == L.stop_count) {
        end = kEndStop;
        break;
      }
      if (left <= L.compact_at) end = kEndCompact;
      V.thr = rec_mn + 1;
      V.tval = rec_mn + 2;
    }
    if (end == kEndEmpty && L.max_levels && levels == L.max_levels) end = kEndLevels;
    // Rows of mostly dead entries are packed: an entry of a row costs its edge's
    // state whether it is alive or not (truss numbers of an R-MAT scale 16 graph:
    // levels 12.1 ms without, 11.0 with; at three quarters 11.3).
    if (kLists && A.pack && left * 2 <= packed) {
      pack_rows(A, gwarp, gwarps);
      packed = left;
      if (!grid_barrier(A.words, A.timeout_ns, crew)) return;
    }
    // The list is rewritten (in order) once an eighth of it is gone, and for
    // the host; dead entries are passed over until then.
    const bool rewrite = end != kEndEmpty || left * 8 <= V.na * 7;
    if (rewrite) {
      uint64_t at = 0;
      for (uint32_t b = threadIdx.x; b < crew.rank; b += blockDim.x) at += ld_relaxed_u64(&kept[b]);
      at = block_sum<uint64_t>(at, wtmp);
      uint32_t* to = L.alive[list ^ 1];
      for (uint64_t j0 = s0; j0 < s1; j0 += blockDim.x) {
        const uint64_t j = j0 + threadIdx.x;
        const uint32_t e = j < s1 ? V.alive[j] : 0u;
        const bool keep = j < s1 && A.state[e] == kAlive && (!L.ngroups || A.gthr[A.egr[e]] != 0);
        uint64_t total;
        const uint64_t p = at + block_excl_scan<uint64_t>(keep ? 1 : 0, wtmp, &total);
        if (keep) to[p] = e;
        at += total;
      }
      list ^= 1;
      V.alive = to;
      V.na = left;
      if (end != kEndEmpty) break;
    }
    if (L.ngroups) {
      if (gtid == 0) *L.tmax = 0;
      if (!grid_barrier(A.words, A.timeout_ns, crew)) return;
      uint32_t top = 0;
      for (uint64_t g = L.group0 + gtid; g < L.group1; g += gthreads) {
        record_group((uint32_t)g, L.gcnt, L.gmin, L.kmax, L.count, L.gthr, L.stop, nkept == 1);
        top = max(top, L.gthr[g]);
      }
      if (top) atomicMax(L.tmax, top);
    }
    // Without a new list or new thresholds nothing was written since the last
    // barrier that the next level reads.
    if (!rewrite && !L.ngroups) continue;
    if (!grid_barrier(A.words, A.timeout_ns, crew)) return;
  }
  flush_tallies(A, tdeg, tdec);
  if (lane_id() == 0 && trec) atomicAdd(&A.acct[2], (unsigned long long)trec);
  if (gtid == 0) {
    LevelsOut* o = L.out;
    o->na = end == kEndEmpty ? 0 : V.na;
    o->rounds = rounds;
    o->count = rec_count;
    o->scanned = scanned;
    o->list = list;
    o->levels = levels;
    o->kept = nkept;
    o->kmax = rec_kmax;
    o->mn = rec_mn;
    o->mx = rec_mx;
    o->recounts = nrec;
    o->r_next = A.r0 + i + 1;
    o->end = end;
    o->gave_up = gave_up;
  }
}

// Host-stepped variant (one launch per round), used when cooperative launch
// is switched off.
__global__ void __launch_bounds__(kPeelThreads) k_level_frontier(PeelArgs A) {
  level_frontier(A, first_level(A), A.r0, A.front[0], &A.cnt[0], (uint64_t)blockIdx.x * blockDim.x + threadIdx.x,
                 (uint64_t)gridDim.x * blockDim.x);
}

__global__ void __launch_bounds__(kPeelThreads) k_round(PeelArgs A, uint32_t i, uint64_t nf) {
  const uint64_t gwarps = ((uint64_t)gridDim.x * blockDim.x) >> 5;
  const uint64_t gwarp = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  uint64_t tdeg = 0, tdec = 0;
  const Level V = first_level(A);
  for (uint64_t f = gwarp; f < nf; f += gwarps)
    peel_edge(A, V, A.front[i & 1][f], A.r0 + i, A.front[(i + 1) & 1], &A.cnt[(i + 1) % 3], tdeg, tdec);
  flush_tallies(A, tdeg, tdec);
}

__global__ void k_peel_init(uint64_t m, uint32_t* __restrict__ state, uint32_t* __restrict__ alive, uint32_t n,
                            const uint64_t* __restrict__ off, uint32_t* __restrict__ adeg) {
  for (uint64_t e = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; e < m; e += (uint64_t)gridDim.x * blockDim.x) {
    state[e] = kAlive;
    alive[e] = (uint32_t)e;
  }
  for (uint64_t v = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; v < n; v += (uint64_t)gridDim.x * blockDim.x)
    adeg[v] = (uint32_t)(off[v + 1] - off[v]);
}

__global__ void k_alive_min(const uint32_t* __restrict__ alive, uint64_t na, const uint32_t* __restrict__ sup,
                            uint32_t* out) {
  uint32_t mn = 0xffffffffu, mx = 0;
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < na; i += (uint64_t)gridDim.x * blockDim.x) {
    const uint32_t s = sup[alive[i]];
    mn = min(mn, s);
    mx = max(mx, s);
  }
  mn = warp_min(mn);
  mx = warp_max(mx);
  if (lane_id() == 0) {
    if (mn != 0xffffffffu) atomicMin(out, mn);
    atomicMax(out + 1, mx);
  }
}

// Per-graph alive edges and minimum support after a level (batched unions).
__global__ void k_track(const uint32_t* __restrict__ alive, uint64_t na, const uint64_t* __restrict__ ends,
                        const uint32_t* __restrict__ sup, const uint32_t* __restrict__ vgid,
                        unsigned long long* __restrict__ gcnt, uint32_t* __restrict__ gmin) {
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < ((na + 31) & ~31ULL);
       i += (uint64_t)gridDim.x * blockDim.x) {
    const bool valid = i < na;
    uint32_t g = 0xffffffffu, sv = 0xffffffffu;
    if (valid) {
      const uint32_t e = alive[i];
      g = vgid[(uint32_t)(ends[e] >> 32)];
      sv = sup[e];
    }
    // Graphs are contiguous in the edge order: aggregate equal graphs.
    const unsigned peers = __match_any_sync(kFull, g);
    const unsigned leader = __ffs(peers) - 1;
    const uint32_t mn = __reduce_min_sync(peers, sv);
    if (valid && lane_id() == leader) {
      atomicAdd(&gcnt[g], (unsigned long long)__popc(peers));
      atomicMin(&gmin[g], mn);
    }
  }
}

// Records every running graph's level and sets its next threshold (its
// minimum support + 1, i.e. level min + 3); a graph with no alive edge, or
// whose first level kept exactly stop[g] edges, is finished (threshold 0).
__global__ void k_track_record(uint32_t ngroups, unsigned long long* __restrict__ gcnt, uint32_t* __restrict__ gmin,
                               uint32_t* __restrict__ kmax, uint64_t* __restrict__ count,
                               uint32_t* __restrict__ gthr, const uint64_t* __restrict__ stop, bool first) {
  for (uint32_t g = blockIdx.x * blockDim.x + threadIdx.x; g < ngroups; g += gridDim.x * blockDim.x)
    record_group(g, gcnt, gmin, kmax, count, gthr, stop, first);
}

__global__ void k_max_u32(const uint32_t* __restrict__ a, uint32_t n, uint32_t* out) {
  uint32_t mx = 0;
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < ((n + 31) & ~31u); i += gridDim.x * blockDim.x)
    mx = max(mx, i < n ? a[i] : 0u);
  mx = warp_max(mx);
  if (lane_id() == 0 && mx) atomicMax(out, mx);
}

__global__ void k_track_init(uint64_t m, const uint64_t* __restrict__ ends, const uint32_t* __restrict__ vgid,
                             uint32_t* __restrict__ egr, uint32_t ngroups, const uint32_t* __restrict__ t0,
                             uint32_t tdef, uint32_t* __restrict__ gthr) {
  for (uint64_t e = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; e < m; e += (uint64_t)gridDim.x * blockDim.x)
    egr[e] = vgid[(uint32_t)(ends[e] >> 32)];
  for (uint32_t g = blockIdx.x * blockDim.x + threadIdx.x; g < ngroups; g += gridDim.x * blockDim.x) {
    const uint32_t t = t0 && t0[g] > 3 ? t0[g] : (tdef > 3 ? tdef : 3);
    gthr[g] = t - 2;
  }
}

// Each team's largest threshold.
__global__ void k_team_tmax(const PeelTeam* __restrict__ teams, uint32_t nteams, const uint32_t* __restrict__ gthr,
                            uint32_t* __restrict__ tmax) {
  const uint32_t t = threadIdx.x;
  if (t >= nteams) return;
  uint32_t mx = 0;
  for (uint32_t g = teams[t].group0; g < teams[t].group1; ++g) mx = max(mx, gthr[g]);
  tmax[t] = mx;
}

__global__ void k_team_keys(uint64_t m, const uint32_t* __restrict__ list, const uint32_t* __restrict__ egr,
                            const uint32_t* __restrict__ team, uint64_t* __restrict__ keys) {
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < m; i += (uint64_t)gridDim.x * blockDim.x)
    keys[i] = team[egr[list[i]]];
}

struct StillAlive {
  const uint32_t* list;
  const uint32_t* state;
  const uint32_t* gthr;  // batched: drop the edges of finished graphs
  const uint32_t* egr;
  __device__ bool keep(uint64_t i) const {
    const uint32_t e = list[i];
    return state[e] == kAlive && (!gthr || gthr[egr[e]] != 0);
  }
  __device__ uint32_t value(uint64_t i) const { return list[i]; }
};

// Ends (u << 32 | v) of the alive edges of a list.
struct AliveEnds {
  const uint32_t* list;
  const uint32_t* state;
  const uint64_t* ends;
  __device__ bool keep(uint64_t i) const { return state[list[i]] == kAlive; }
  __device__ uint64_t value(uint64_t i) const { return ends[list[i]]; }
};

// Peel state of one working graph on the device.
struct Peeler {
  Ctx* c;
  const Sub* s;
  uint32_t* sup;
  uint32_t* truss;
  DBuf state, alive[2], front[2], cnt, out, mm, adeg, acct, table, big;
  DBuf rows_len, rows_adj, rows_eid;  // list mode: PeelArgs::rlen, radj, reid
  uint32_t table_bits = 0;
  uint64_t scanned = 0;  // alive-list entries scanned by level frontiers
  int ai = 0;
  uint64_t na = 0;
  uint32_t r = 1;  // next round number
  uint64_t fail_below = 0;  // set while a level is tried from a snapshot (PeelArgs::fail_below)
  unsigned coop_grid = 0;
  unsigned threads = kLevelThreads;  // of a k_levels block
  size_t smem = 0;
  PeelResult* res;

  void init() {
    const uint64_t m = s->m;
    state = DBuf(c, m * sizeof(uint32_t));
    alive[0] = DBuf(c, m * sizeof(uint32_t));
    alive[1] = DBuf(c, m * sizeof(uint32_t));
    front[0] = DBuf(c, m * sizeof(uint32_t));
    front[1] = DBuf(c, m * sizeof(uint32_t));
    cnt = DBuf(c, (kCounters + kMaxGrid) * sizeof(unsigned long long));
    out = DBuf(c, sizeof(LevelsOut));
    mm = DBuf(c, 8);
    adeg = DBuf(c, ((uint64_t)s->n + 1) * sizeof(uint32_t));
    if (!acct.get()) {
      acct = DBuf(c, 4 * sizeof(unsigned long long));
      zero(c, acct.get(), acct.bytes());
    }
    ai = 0;
    k_peel_init<<<grid_for(std::max<uint64_t>(m, s->n), 256, c->num_sms * 16), 256, 0, c->stream>>>(
        m, state.as<uint32_t>(), alive[0].as<uint32_t>(), s->n, s->off.as<uint64_t>(), adeg.as<uint32_t>());
    // Dense mode: keep the alive list in tile order (compaction preserves it).
    if (s->W)
      KT_CUDA(cudaMemcpyAsync(alive[0].get(), s->order.get(), m * sizeof(uint32_t), cudaMemcpyDeviceToDevice,
                              c->stream));
    KT_LAUNCHED(c);
    na = m;
    coop_grid = 0;
    build_table();
    if (c->opt.persistent || s->W) {
      allow_max_dynamic_smem(kernel());
      // The threads of a block that leave most warps on an SM beside the rows'
      // shared memory, the larger number where they are equal.  (Beyond some 1,700
      // words one block of 512 would fit, three of 256 or seven of 128, and a round of
      // decrements waits for its chains of accesses: 36M edges on 60,000 vertices
      // 2,493 ms with 16 warps, 1,730 with 24, 1,530 with 28.)
      int per_sm = 0;
      const unsigned widest = s->W < kWideRow ? kLevelThreads : kLevelThreads / 2;
      const unsigned most = s->W < kWideRow ? 2 * kLevelThreads : 5 * (kLevelThreads / 2);  // by registers
      threads = 0;
      for (unsigned t = widest; t >= 128 && per_sm * threads < most; t /= 2) {
        const size_t want = table.get() ? sizeof(RowBatch) : s->W <= kShortRow ? 0 : dense_smem_bytes(s->W, t);
        if (t > 128 && want > kRowsSmem) continue;
        int fit = 0;
        KT_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&fit, kernel(), (int)t, want));
        if (threads && fit * t <= per_sm * threads) continue;
        per_sm = fit;
        threads = t;
        smem = want;
      }
      // A warp counts eight edges at once, or looks up kJobWide entries a lane.
      coop_grid = coop_blocks_for(std::min(coop_blocks(c, per_sm), kMaxGrid), s->m, threads / 4);
    }
  }

  const void* kernel() const {
    if (table.get()) return (const void*)k_levels<true, false, kLevelThreads, 2>;
    if (!teams.empty()) return (const void*)k_levels<false, true, kLevelThreads, 2>;
    return s->W < kWideRow ? (const void*)k_levels<false, false, kLevelThreads, 2>
                           : (const void*)k_levels<false, false, kLevelThreads / 2, 5>;
  }

  // List mode: the edge hash table, 8 to 20 bytes an edge, when the budget
  // has room for it (else, and in host-stepped rounds, rows are merged).
  void build_table() {
    table.release();
    big.release();
    rows_len.release();
    rows_adj.release();
    rows_eid.release();
    if (s->W || !c->opt.persistent) return;
    table_bits = 10;
    while (table_bits < 32 && (2ull << table_bits) < 5 * s->m) ++table_bits;
    const uint64_t bytes = (8ull << table_bits) + (s->m + s->n) * sizeof(uint32_t);
    // (Beside it, what the levels may ask for later: snapshots, a rebuilt graph.)
    const uint64_t later = (truss ? 0 : 32 * s->m) + (1u << 20);
    if ((2ull << table_bits) < 5 * s->m || (c->budget && c->in_use + bytes + later > c->budget)) return;
    if (!big.try_alloc(c, s->m * sizeof(uint32_t)) || !rows_len.try_alloc(c, s->n * sizeof(uint32_t)) ||
        !table.try_alloc(c, 8ull << table_bits))
      return;
    KT_CUDA(cudaMemsetAsync(table.get(), 0xff, 8ull << table_bits, c->stream));
    k_table_build<<<grid_for(s->m, 256, c->num_sms * 16), 256, 0, c->stream>>>(
        s->m, s->ends.as<uint64_t>(), table.as<unsigned long long>(), table_bits);
    KT_LAUNCHED(c);
    k_row_lengths<<<grid_for(s->n, 256, c->num_sms * 16), 256, 0, c->stream>>>(s->off.as<uint64_t>(), s->n,
                                                                             rows_len.as<uint32_t>());
    KT_LAUNCHED(c);
    // Rows that may be packed, when every level is peeled and there is room for
    // a copy.
    const uint64_t rows = 2 * s->m * sizeof(uint32_t);
    if (!truss || (c->budget && c->in_use + 2 * rows + (1u << 20) > c->budget)) return;
    if (!rows_adj.try_alloc(c, rows) || !rows_eid.try_alloc(c, rows)) {
      rows_adj.release();
      return;
    }
    lower_ids(c, *s);
    KT_CUDA(cudaMemcpyAsync(rows_adj.get(), s->adj.get(), rows, cudaMemcpyDeviceToDevice, c->stream));
    KT_CUDA(cudaMemcpyAsync(rows_eid.get(), s->eid.get(), rows, cudaMemcpyDeviceToDevice, c->stream));
  }

  PeelArgs args(uint32_t t) {
    PeelArgs A;
    A.ends = s->ends.as<uint64_t>();
    A.off = s->off.as<uint64_t>();
    A.adj = s->adj.as<uint32_t>();
    lower_ids(c, *s);
    A.eid = s->eid.as<uint32_t>();
    A.sup = sup;
    A.state = state.as<uint32_t>();
    A.truss = truss;
    A.alive = alive[ai].as<uint32_t>();
    A.na = na;
    A.front[0] = front[0].as<uint32_t>();
    A.front[1] = front[1].as<uint32_t>();
    A.cnt = cnt.as<unsigned long long>();
    A.cap = s->m;
    A.thr = t - 2;
    A.tval = t - 1;
    A.r0 = r;
    A.adeg = adeg.as<uint32_t>();
    A.acct = acct.as<unsigned long long>();
    A.R = s->W ? dense_rows(*s) : DenseRows{nullptr, 0, nullptr, nullptr, nullptr, nullptr, nullptr};
    if (!c->opt.peel_bitset) A.R.sbits = nullptr;
    A.wavg = s->W ? (float)((double)s->bit_words / std::max<uint32_t>(s->n, 1)) : 0.f;
    A.bit_words = s->W ? s->bit_words : 0;
    A.gamma = (uint32_t)std::max<int64_t>(1, c->opt.recount_gamma);
    A.search_ratio = (uint32_t)std::min<int64_t>(std::max<int64_t>(1, c->opt.peel_search_ratio), 1 << 20);
    A.split = (uint32_t)std::min<int64_t>(std::max<int64_t>(0, c->opt.peel_split), 1 << 14);  // units fit 32 bits
    A.words = dev_words(c);
    A.timeout_ns = (unsigned long long)c->opt.timeout_ms * 1000000ULL;
    A.gthr = track ? gthr.as<uint32_t>() : nullptr;
    A.egr = track ? egr.as<uint32_t>() : nullptr;
    A.gthr_max = track ? tmax.as<uint32_t>() : nullptr;
    A.table = table.as<unsigned long long>();
    A.table_bits = table_bits;
    A.big = big.as<uint32_t>();
    A.n = s->n;
    A.pack = rows_adj.get() && !fail_below;  // (a level tried may be undone)
    A.radj = rows_adj.get() ? rows_adj.as<uint32_t>() : s->adj.as<uint32_t>();
    A.reid = rows_eid.get() ? rows_eid.as<uint32_t>() : s->eid.as<uint32_t>();
    A.rlen = rows_len.as<uint32_t>();
    A.fail_below = fail_below;
    return A;
  }

  // A level tried from a snapshot: the cascade gives up once its truss can
  // no longer hold t(t-1)/2 edges.
  uint64_t try_level(uint32_t t) {
    fail_below = (uint64_t)t * (t - 1) / 2;
    const uint64_t left = cascade(t);
    fail_below = 0;
    return left;
  }

  // Levels from t up on the device (coop_grid): see LevelsArgs for when it
  // ends.  The alive list, na and r are the last level's.
  LevelsOut levels(uint32_t t, uint32_t max_levels, uint64_t stop_count, uint64_t compact_at) {
    PeelArgs A = args(t);
    LevelsArgs L{};
    L.alive[0] = alive[ai].as<uint32_t>();
    L.alive[1] = alive[ai ^ 1].as<uint32_t>();
    L.max_levels = max_levels;
    L.stop_count = stop_count;
    L.compact_at = compact_at;
    L.out = out.as<LevelsOut>();
    if (track) {
      L.ngroups = track->ngroups;
      L.gcnt = tcnt.as<unsigned long long>();
      L.gmin = tmin.as<uint32_t>();
      L.kmax = track->kmax;
      L.count = track->count;
      L.gthr = gthr.as<uint32_t>();
      L.tmax = tmax.as<uint32_t>();
      L.stop = track->stop;
      L.group1 = track->ngroups;
    }
    if (!teams.empty()) {
      L.teams = dteams.as<PeelTeam>();
      L.nteams = (uint32_t)teams.size();
      L.counters = kCounters + coop_grid;
      L.team_words = team_words.as<DevWords>();
    }
    zero(c, cnt.get(), teams.empty() ? kCounters * sizeof(unsigned long long) : cnt.bytes());
    cudaEvent_t e0;
    c->timer.begin(c->stream, &c->stats.ms_peel_kernel, &e0);
    const auto t_start = std::chrono::steady_clock::now();
    const uint64_t before = na;
    LevelsOut h;
    {
      CoopLock coop(c);
      void* p[] = {&A, &L};
      KT_CUDA(cudaLaunchCooperativeKernel(kernel(), dim3(teams.empty() ? coop_grid : team_blocks(teams)), dim3(threads),
                                          p, smem, c->stream));
      KT_LAUNCHED(c);
      c->timer.end(c->stream, e0, &c->stats.ms_peel_kernel);
      if (teams.empty()) {
        read_checked(c, &h, out.get(), sizeof(h), "truss peel");
      } else {
        merge_team_errors(c, team_words.get(), (uint32_t)teams.size());
        LevelsOut each[kMaxPeelTeams];
        static_assert(sizeof(each) <= 3072, "read through the context's pinned words");
        read_checked(c, each, out.get(), teams.size() * sizeof(LevelsOut), "truss peel");
        h = each[0];
        for (size_t i = 1; i < teams.size(); ++i) {  // the most of each; every team ends empty
          h.rounds = std::max(h.rounds, each[i].rounds);
          h.levels = std::max(h.levels, each[i].levels);
          h.r_next = std::max(h.r_next, each[i].r_next);
          h.scanned += each[i].scanned;
          h.recounts += each[i].recounts;
        }
      }
    }
    c->stats.peel_launches++;
    KT_LOG(c,
           "kt: levels from %u on %llu alive of %llu edges (n %u, W %u): %u levels, %llu rounds (%u recount), "
           "%llu left%s, %.3f ms\n",
           t, (unsigned long long)before, (unsigned long long)s->m, s->n, s->W, h.levels,
           (unsigned long long)h.rounds, h.recounts, (unsigned long long)h.na, h.gave_up ? ", gave up" : "",
           std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now() - t_start).count());
    r = h.r_next;
    scanned += h.scanned;
    res->rounds += h.rounds;
    res->levels += h.levels;
    if (h.end != kEndEmpty) {
      na = h.na;
      mn_left = h.mn;
      mx_left = h.mx;
      if (h.list) ai ^= 1;
    }
    return h;
  }

  // Removes every alive edge with support < t-2, to the fixpoint; returns
  // the alive count.
  uint64_t cascade(uint32_t t) {
    if (coop_grid) {
      const LevelsOut h = levels(t, 1, 0, 0);
      if (h.end == kEndEmpty && !h.gave_up) na = 0;
      return h.end == kEndEmpty ? 0 : na;
    }
    PeelArgs A = args(t);
    zero(c, cnt.get(), kCounters * sizeof(unsigned long long));
    cudaEvent_t e0;
    c->timer.begin(c->stream, &c->stats.ms_peel_kernel, &e0);
    uint64_t rounds = 0;
    bool gave_up = false;
    scanned += na;
    {
      k_level_frontier<<<grid_for(na, kPeelThreads, c->num_sms * 16), kPeelThreads, 0, c->stream>>>(A);
      KT_LAUNCHED(c);
      uint64_t left = na;
      for (uint32_t i = 0;; ++i) {
        const uint64_t nf = read_word<unsigned long long>(c, A.cnt + (i % 3));
        if (nf == 0) break;
        if (left - nf < A.fail_below) {
          gave_up = true;
          break;
        }
        left -= nf;
        ++rounds;
        KT_CUDA(cudaMemsetAsync(A.cnt + ((i + 1) % 3), 0, sizeof(unsigned long long), c->stream));
        k_round<<<grid_for(nf * 32, kPeelThreads, c->num_sms * 16), kPeelThreads, 0, c->stream>>>(A, i, nf);
        KT_LAUNCHED(c);
      }
    }
    c->timer.end(c->stream, e0, &c->stats.ms_peel_kernel);
    c->stats.peel_launches++;
    check_words(c, "truss peel");
    KT_LOG(c, "kt: cascade level %u: %llu alive of %llu edges (n %u), %llu rounds%s\n", t, (unsigned long long)na,
           (unsigned long long)s->m, s->n, (unsigned long long)rounds, gave_up ? ", gave up" : "");
    r += (uint32_t)rounds + 1;
    res->rounds += rounds;
    res->levels++;
    if (gave_up) return 0;  // the level is empty; the state is partial and the caller undoes it
    na = compact(c, na,
                 StillAlive{alive[ai].as<uint32_t>(), state.as<uint32_t>(), A.gthr, A.egr},
                 alive[ai ^ 1].as<uint32_t>());
    ai ^= 1;
    return na;
  }

  // Algorithmic bytes of this peel: 8 per alive-degree unit of every deleted
  // edge (neighbour id + edge id), 8 per support decrement (read-modify-
  // write), 4 per alive-list entry scanned by a level frontier.  The dense
  // recount rounds' bitset rows (4 W bytes per recounted edge, mostly from
  // L2) are kept apart in peel_recount_bytes.
  void account() {
    uint64_t h[3];
    copy_d2h(c, h, acct.get(), 24);
    const double wavg = s->W ? (double)s->bit_words / std::max<uint32_t>(s->n, 1) : 0.0;
    c->stats.peel_bytes += 8 * h[0] + 8 * h[1] + 4 * scanned;
    c->stats.peel_recount_bytes += (uint64_t)(4.0 * wavg * (double)h[2]);
    c->stats.peel_decrements += h[1];
  }

  // Batched unions: per-graph thresholds and records after a level.
  const GraphTrack* track = nullptr;
  DBuf tcnt, tmin, gthr, egr, tmax;
  void init_track(uint32_t t0) {
    const uint32_t G = std::max<uint32_t>(track->ngroups, 1);
    tcnt = DBuf(c, (uint64_t)G * 8);
    tmin = DBuf(c, (uint64_t)G * 4);
    gthr = DBuf(c, (uint64_t)G * 4);
    egr = DBuf(c, s->m * 4);
    tmax = DBuf(c, 4);
    zero(c, tcnt.get(), tcnt.bytes());
    KT_CUDA(cudaMemsetAsync(tmin.get(), 0xff, tmin.bytes(), c->stream));
    k_track_init<<<grid_for(std::max<uint64_t>(s->m, G), 256, c->num_sms * 16), 256, 0, c->stream>>>(
        s->m, s->ends.as<uint64_t>(), track->vgid, egr.as<uint32_t>(), track->ngroups, track->t0, t0,
        gthr.as<uint32_t>());
    KT_LAUNCHED(c);
    update_tmax();
  }
  // Teams for the levels of a union with bitset rows of at most kShortRow words:
  // its alive list is put in their order, where the sort of it has room.  (With
  // longer rows the recounts of a graph are bound by bandwidth, of which a team
  // has its share only: 7.3M edges, rows of up to 196 words, 9.4 ms in step and
  // 10.9 by teams; 3.9M edges, rows of up to 44 words, 15.1 and 10.7.)
  std::vector<TeamSpan> teams;
  DBuf dteams, team_words;
  void init_teams() {
    constexpr uint64_t kLeastEdges = 1u << 19;  // (smaller unions are no faster by teams)
    const size_t G = s->group_n.size();
    if (!s->W || s->W > kShortRow || !s->roff.get() || G != track->ngroups || s->m < kLeastEdges) return;
    DBuf room;  // for the sort
    if ((c->budget && c->in_use + 40 * s->m > c->budget) || !room.try_alloc(c, 24 * s->m)) return;
    room.release();
    std::vector<uint64_t> starts(G + 1, 0), words(G + 1, 0);
    for (size_t g = 0; g < G; ++g) {
      starts[g + 1] = starts[g] + s->group_n[g];
      words[g + 1] = words[g] + (uint64_t)s->group_n[g] * (((s->group_n[g] + 31) / 32 + 3) & ~3u);
    }
    const std::vector<uint64_t> at = gather_offsets(c, s->off.as<uint64_t>(), starts);
    const void* by_teams = (const void*)k_levels<false, true, kLevelThreads, 2>;
    allow_max_dynamic_smem(by_teams);
    int per_sm = 0;
    KT_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, by_teams, (int)threads, smem));
    if (per_sm < 1) return;
    teams = split_teams(at, kMaxPeelTeams, std::min(coop_grid, coop_blocks(c, per_sm)));
    if (teams.empty()) return;
    std::vector<PeelTeam> t;
    std::vector<uint32_t> of(G);  // each graph's team
    for (const TeamSpan& x : teams) {
      for (uint64_t g = x.first; g < x.last; ++g) of[g] = (uint32_t)t.size();
      const uint64_t w = words[x.last] - words[x.first], n = starts[x.last] - starts[x.first];
      t.push_back(PeelTeam{x.block0, x.blocks, (uint32_t)x.first, (uint32_t)x.last, at[x.first] / 2,
                           (at[x.last] - at[x.first]) / 2, words[x.first], w,
                           (float)((double)w / std::max<uint64_t>(n, 1))});
    }
    dteams = DBuf(c, t.size() * sizeof(PeelTeam));
    copy_h2d(c, dteams.get(), t.data(), t.size() * sizeof(PeelTeam));
    team_words = DBuf(c, t.size() * sizeof(DevWords));
    zero(c, team_words.get(), team_words.bytes());
    out = DBuf(c, t.size() * sizeof(LevelsOut));
    cnt = DBuf(c, t.size() * (kCounters + coop_grid) * sizeof(unsigned long long));
    tmax = DBuf(c, t.size() * sizeof(uint32_t));
    k_team_tmax<<<1, kMaxPeelTeams, 0, c->stream>>>(dteams.as<PeelTeam>(), (uint32_t)t.size(), gthr.as<uint32_t>(),
                                                   tmax.as<uint32_t>());
    KT_LAUNCHED(c);
    DBuf dof(c, G * sizeof(uint32_t)), keys(c, s->m * sizeof(uint64_t));
    copy_h2d(c, dof.get(), of.data(), G * sizeof(uint32_t));
    k_team_keys<<<grid_for(s->m, 256, c->num_sms * 16), 256, 0, c->stream>>>(
        s->m, alive[ai].as<uint32_t>(), egr.as<uint32_t>(), dof.as<uint32_t>(), keys.as<uint64_t>());
    KT_LAUNCHED(c);
    radix_sort_u64(c, keys.as<uint64_t>(), alive[ai].as<uint32_t>(), s->m, {{0, bits_for(t.size())}});
  }

  void update_tmax() {
    zero(c, tmax.get(), 4);
    k_max_u32<<<grid_for(track->ngroups, 256, c->num_sms * 4), 256, 0, c->stream>>>(
        gthr.as<uint32_t>(), track->ngroups, tmax.as<uint32_t>());
    KT_LAUNCHED(c);
  }
  void record_groups(bool first) {
    if (na) {
      k_track<<<grid_for(na, 256, c->num_sms * 16), 256, 0, c->stream>>>(
          alive[ai].as<uint32_t>(), na, s->ends.as<uint64_t>(), sup, track->vgid, tcnt.as<unsigned long long>(),
          tmin.as<uint32_t>());
      KT_LAUNCHED(c);
    }
    k_track_record<<<grid_for(track->ngroups, 256, c->num_sms * 4), 256, 0, c->stream>>>(
        track->ngroups, tcnt.as<unsigned long long>(), tmin.as<uint32_t>(), track->kmax, track->count,
        gthr.as<uint32_t>(), track->stop, first);
    KT_LAUNCHED(c);
    update_tmax();
  }

  // Replaces the working graph by its alive part (renumbered, with its own
  // bitsets and exact supports) once most edges are gone; the alive edges
  // form a truss, so their supports in the new graph equal their current
  // ones.  Returns whether it compacted.
  uint64_t compact_at() const { return truss || track || s->m < (1u << 20) ? 0 : s->m / 4; }
  bool compact_graph(std::unique_ptr<Sub>& own, DBuf& own_sup) {
    if (na == 0 || na > compact_at()) return false;
    account();
    zero(c, acct.get(), acct.bytes());
    scanned = 0;
    DBuf keys(c, na * sizeof(uint64_t));
    const uint64_t k = kt::compact(c, na, AliveEnds{alive[ai].as<uint32_t>(), state.as<uint32_t>(),
                                                    s->ends.as<uint64_t>()},
                                   keys.as<uint64_t>());
    std::unique_ptr<Sub> ns(new Sub);
    // The alive list is in edge-id order unless the graph has bitsets (tile
    // order), so its ends are already sorted then.
    build_sub_from_keys(c, keys.as<uint64_t>(), k, s->n, *ns, s->W == 0);
    DBuf nsup(c, (ns->m ? ns->m : 1) * sizeof(uint32_t));
    edge_support(c, *ns, nsup.as<uint32_t>());
    own.swap(ns);
    own_sup = std::move(nsup);
    s = own.get();
    sup = own_sup.as<uint32_t>();
    init();
    return true;
  }

  // Finds the top level by bisection, between lo (the current state is the
  // lo-truss, non-empty) and hi (the hi-truss is empty): a level whose truss
  // is empty is undone from a snapshot of the state (supports, edge states,
  // alive degrees, bitsets; the alive list of the snapshot stays in the
  // other buffer), a non-empty one is kept.  A t-truss is non-empty exactly
  // for t <= kmax, so this ends with res at kmax and its edge count.
  void bisect(uint32_t lo, uint32_t hi, PeelResult& out) {
    DBuf ssup(c, s->m * sizeof(uint32_t)), sstate(c, s->m * sizeof(uint32_t)), sdeg(c, adeg.bytes()), sbits;
    if (s->W) sbits.alloc(c, s->bits.bytes());
    uint64_t na0 = 0;
    int ai0 = 0;
    auto copy = [&](void* dst, const void* src, size_t bytes) {
      KT_CUDA(cudaMemcpyAsync(dst, src, bytes, cudaMemcpyDeviceToDevice, c->stream));
    };
    auto save = [&] {
      copy(ssup.get(), sup, s->m * sizeof(uint32_t));
      copy(sstate.get(), state.get(), s->m * sizeof(uint32_t));
      copy(sdeg.get(), adeg.get(), adeg.bytes());
      if (s->W) copy(sbits.get(), s->bits.get(), s->bits.bytes());
      na0 = na;
      ai0 = ai;
    };
    save();
    while (hi - lo > 1) {
      const uint32_t mid = lo + (hi - lo) / 2;
      const uint64_t left = try_level(mid);
      if (left) {
        uint32_t mn, mx;
        minmax(mn, mx);
        lo = mn + 2;  // >= mid
        out.kmax = lo;
        out.count = left;
        if (hi - lo > 1) save();
      } else {
        copy(sup, ssup.get(), s->m * sizeof(uint32_t));
        copy(state.get(), sstate.get(), s->m * sizeof(uint32_t));
        copy(adeg.get(), sdeg.get(), adeg.bytes());
        if (s->W) copy(s->bits.get(), sbits.get(), s->bits.bytes());
        na = na0;
        ai = ai0;
        hi = mid;
      }
    }
    KT_LOG(c, "kt: bisection ends at level %u with %llu edges\n", out.kmax, (unsigned long long)out.count);
  }

  // (min, max) support over alive edges, after a level that left some.
  uint32_t mn_left = 0, mx_left = 0;  // on the device: found with the level
  void minmax(uint32_t& mn, uint32_t& mx) {
    if (coop_grid) {
      mn = mn_left;
      mx = mx_left;
      return;
    }
    const uint32_t init[2] = {0xffffffffu, 0u};
    copy_h2d(c, mm.get(), init, 8);
    k_alive_min<<<grid_for(na, 256, c->num_sms * 8), 256, 0, c->stream>>>(alive[ai].as<uint32_t>(), na, sup,
                                                                            mm.as<uint32_t>());
    KT_LAUNCHED(c);
    uint32_t h[2];
    copy_d2h(c, h, mm.get(), 8);
    mn = h[0];
    mx = h[1];
  }
};

}  // namespace

void build_sub_from_keys(Ctx* c, uint64_t* keys, uint64_t m, uint32_t n_ids, Sub& out, bool sorted) {
  Graph g;
  build_graph(c, keys, m, n_ids, g, false, sorted);
  build_sub_all(c, g, out);
}

PeelResult truss_peel(Ctx* c, const Sub& s, uint32_t* sup, uint32_t t0, uint64_t stop_count, uint32_t* truss,
                      uint32_t guess, const GraphTrack* track) {
  PeelResult res;
  if (s.m == 0) return res;
  if (t0 < 3) t0 = 3;
  std::unique_ptr<Sub> own;
  DBuf own_sup;
  Peeler P{c, &s, sup, truss};
  P.res = &res;
  P.track = track;
  P.init();
  uint32_t t = t0;
  if (track) {
    // Batched: every graph climbs its own levels (min-support jumps, its own
    // first level and early stop); a cascade runs all of them at once.
    if (track->ngroups == 0) return res;
    P.init_track(t0);
    if (P.coop_grid) {
      P.init_teams();
      P.levels(t, 0, 0, 0);
      P.account();
      return res;
    }
    for (bool first = true; P.na; first = false) {
      P.cascade(t);
      P.record_groups(first);
    }
    P.account();
    return res;
  }
  // Jump phase: try `guess` (> t0) from a snapshot; halve toward t0 on failure.
  if (!truss && guess > t0) {
    DBuf snap_sup(c, s.m * sizeof(uint32_t)), snap_state(c, s.m * sizeof(uint32_t));
    DBuf snap_deg(c, P.adeg.bytes());
    DBuf snap_bits;
    if (s.W) {
      snap_bits.alloc(c, s.bits.bytes());
      KT_CUDA(cudaMemcpyAsync(snap_bits.get(), s.bits.get(), s.bits.bytes(), cudaMemcpyDeviceToDevice, c->stream));
    }
    KT_CUDA(cudaMemcpyAsync(snap_deg.get(), P.adeg.get(), P.adeg.bytes(), cudaMemcpyDeviceToDevice, c->stream));
    KT_CUDA(cudaMemcpyAsync(snap_sup.get(), sup, s.m * sizeof(uint32_t), cudaMemcpyDeviceToDevice, c->stream));
    KT_CUDA(cudaMemcpyAsync(snap_state.get(), P.state.get(), s.m * sizeof(uint32_t), cudaMemcpyDeviceToDevice,
                            c->stream));
    const uint64_t na0 = P.na;
    const int ai0 = P.ai;
    uint32_t g = guess;
    while (g > t0) {
      if (P.try_level(g)) {
        t = g;
        break;
      }
      // Undo: the alive list of the snapshot is still in the other buffer.
      KT_CUDA(cudaMemcpyAsync(sup, snap_sup.get(), s.m * sizeof(uint32_t), cudaMemcpyDeviceToDevice, c->stream));
      KT_CUDA(cudaMemcpyAsync(P.state.get(), snap_state.get(), s.m * sizeof(uint32_t), cudaMemcpyDeviceToDevice,
                              c->stream));
      KT_CUDA(cudaMemcpyAsync(P.adeg.get(), snap_deg.get(), P.adeg.bytes(), cudaMemcpyDeviceToDevice, c->stream));
      if (s.W)
        KT_CUDA(cudaMemcpyAsync(s.bits.get(), snap_bits.get(), s.bits.bytes(), cudaMemcpyDeviceToDevice, c->stream));
      P.ai = ai0;
      P.na = na0;
      g = t0 + (g - t0) / 2;
    }
    if (t != t0) {
      // The t-truss is non-empty: continue upward from it.
      uint32_t mn, mx;
      P.minmax(mn, mx);
      res.kmax = mn + 2;
      res.count = P.na;
      t = mn + 3;
      stop_count = 0;
    }
  }
  // Levels climbed one at a time before a long climb turns into a bisection
  // (peel_bisect_after, 0 = never), and the gap to the support bound that
  // makes it one (peel_bisect_gap).
  const uint64_t bisect_after = (uint64_t)std::max<int64_t>(0, c->opt.peel_bisect_after);
  const uint64_t bisect_gap = (uint64_t)std::max<int64_t>(1, c->opt.peel_bisect_gap);
  bool first = true;
  uint32_t climbed = 0;
  while (true) {
    uint32_t mn, mx;
    if (P.coop_grid) {
      // All levels up to the next thing to do here.
      const bool climbing = !truss && bisect_after && climbed < bisect_after;
      const LevelsOut h = P.levels(t, climbing ? (uint32_t)(bisect_after - climbed) : 0, first ? stop_count : 0,
                                   P.compact_at());
      if (h.kept) {
        res.kmax = h.kmax;
        res.count = h.count;
      }
      if (h.end == kEndEmpty) break;
      if (h.end == kEndStop) {
        res.kmax = t;
        res.stopped_early = true;
        P.account();
        return res;
      }
      climbed += h.kept;
      mn = h.mn;
      mx = h.mx;
    } else {
      const uint64_t left = P.cascade(t);
      if (left == 0) break;
      if (first && stop_count && left == stop_count) {
        res.kmax = t;
        res.count = left;
        res.stopped_early = true;
        P.account();
        return res;
      }
      P.minmax(mn, mx);
      res.kmax = mn + 2;
      res.count = left;
      ++climbed;
    }
    first = false;
    t = mn + 3;
    P.compact_graph(own, own_sup);
    if (!truss && bisect_after && climbed == bisect_after) {
      // No level above the support bound of the alive edges is non-empty
      // (removed edges keep supports below the current level's threshold).
      const uint32_t ub = support_bound(c, P.sup, P.s->m, mx + 2);
      if (ub >= t + bisect_gap) {
        KT_LOG(c, "kt: level %u, support bound %u: bisecting\n", t, ub);
        P.bisect(res.kmax, ub + 1, res);
        break;
      }
    }
  }
  if (res.kmax < 3) {
    res.kmax = 0;
    res.count = 0;
  }
  P.account();
  return res;
}

}  // namespace kt
