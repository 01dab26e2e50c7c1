// Stage (c): k-core peeling on the full graph.
//
// A probe peels the current vertex set to its k-core: the vertices of degree
// < k form the first frontier, and each round removes the frontier and
// decrements the degrees of its surviving neighbours; a neighbour whose
// degree steps from k to k-1 (atomicSub returns k) joins the next frontier,
// so every vertex enters a frontier at most once.  The whole search runs in
// one cooperative launch (k_core_search), which ends early only for a
// compaction.  Rows of more than kcore_big_row (option, 512) entries are cut
// into windows dealt to every warp of the grid, so hub rows do not serialise on
// one warp.
//
// The search for the maximum core (the reference steps k by a fixed stride
// with host backups, src/kc.cu:770-884) ramps k geometrically from the
// current core (each success is permanent; removed vertices keep the probe's
// tag), then bisects; a probe that empties the graph is undone by reviving
// its tag and copying the degrees before it back.  The tags of successful probes increase
// with their level, which lets any lower core be restored later without a
// snapshot: revive the vertices whose tag is newer than the last probe at or
// below that level, recount degrees, and probe once more; below a compacted
// copy, in the graph that it was made from, which keeps its tags.
#include <algorithm>
#include <chrono>
#include <cmath>
#include <cstdio>
#include <cstring>

#include "compact.cuh"
#include "kcore.h"
#include "rows.cuh"
#include "teams.h"

namespace kt {
namespace {

struct AliveF {
  const uint32_t* rem;
  __device__ bool keep(uint64_t v) const { return rem[v] == kAlive; }
  __device__ uint32_t value(uint64_t v) const { return (uint32_t)v; }
};

__global__ void k_init_state(const uint32_t* __restrict__ deg0, uint64_t n, uint32_t* __restrict__ deg,
                             uint32_t* __restrict__ rem) {
  for (uint64_t v = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; v < n; v += (uint64_t)gridDim.x * blockDim.x) {
    const uint32_t d = deg0[v];
    deg[v] = d;
    rem[v] = d ? kAlive : 0u;  // isolated vertices leave at tag 0 (level 1)
  }
}

// Warp-aggregated push of `want` lanes into list[cnt...].  Called by the whole
// warp.
__device__ __forceinline__ void push_warp(bool want, uint32_t item, uint32_t* list, unsigned long long* cnt,
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

__global__ void k_frontier_init(const uint32_t* __restrict__ alive, uint64_t n_alive, const uint32_t* __restrict__ deg,
                                uint32_t* __restrict__ rem, uint32_t k, uint32_t tag, uint32_t* __restrict__ front,
                                unsigned long long* fcnt, uint64_t cap, uint32_t* err) {
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < ((n_alive + 31) & ~31ULL);
       i += (uint64_t)gridDim.x * blockDim.x) {
    bool want = false;
    uint32_t v = 0;
    if (i < n_alive) {
      v = alive[i];
      if (rem[v] == kAlive && deg[v] < k) {
        rem[v] = tag;
        want = true;
      }
    }
    push_warp(want, v, front, fcnt, cap, err);
  }
}

// Removes the frontier: warp per vertex; rows longer than big_row go to the
// big list for k_expand_big.
__global__ void k_expand(const uint32_t* __restrict__ front, uint64_t nf, const uint64_t* __restrict__ off,
                         const uint32_t* __restrict__ adj, uint32_t* __restrict__ deg, uint32_t* __restrict__ rem,
                         uint32_t k, uint32_t tag, uint32_t* __restrict__ next, unsigned long long* ncnt,
                         uint32_t* __restrict__ big, unsigned long long* nbig, uint64_t cap, uint32_t* err,
                         uint32_t big_row) {
  const uint64_t warps = (uint64_t)gridDim.x * (blockDim.x >> 5);
  for (uint64_t f = (uint64_t)blockIdx.x * (blockDim.x >> 5) + warp_id(); f < nf; f += warps) {
    const uint32_t v = front[f];
    const uint64_t b = off[v], e = off[v + 1];
    if (e - b > big_row) {
      if (lane_id() == 0) {
        const unsigned long long p = atomicAdd(nbig, 1ULL);
        if (p < cap)
          big[p] = v;
        else
          atomicOr(err, kDevErrCapacity);
      }
      continue;
    }
    for (uint64_t j = b + lane_id(); j < ((e - b + 31) & ~31ULL) + b; j += 32) {
      bool want = false;
      uint32_t w = 0;
      if (j < e) {
        w = adj[j];
        if (rem[w] == kAlive) {
          const uint32_t old = atomicSub(&deg[w], 1u);
          if (old == k) {
            rem[w] = tag;
            want = true;
          }
        }
      }
      push_warp(want, w, next, ncnt, cap, err);
    }
  }
}

// Big rows: one block per row (rows round-robin over blocks), each warp
// taking 32-entry windows of it.
__global__ void k_expand_big(const uint32_t* __restrict__ big, const unsigned long long* nbig_p,
                             const uint64_t* __restrict__ off, const uint32_t* __restrict__ adj,
                             uint32_t* __restrict__ deg, uint32_t* __restrict__ rem, uint32_t k, uint32_t tag,
                             uint32_t* __restrict__ next, unsigned long long* ncnt, uint64_t cap, uint32_t* err) {
  const uint64_t nbig = *nbig_p;
  for (uint64_t bi = blockIdx.x; bi < nbig; bi += gridDim.x) {
    const uint32_t v = big[bi];
    const uint64_t b = off[v], e = off[v + 1];
    for (uint64_t j0 = b + warp_id() * 32; j0 < e; j0 += blockDim.x) {
      const uint64_t j = j0 + lane_id();
      bool want = false;
      uint32_t w = 0;
      if (j < e) {
        w = adj[j];
        if (rem[w] == kAlive) {
          const uint32_t old = atomicSub(&deg[w], 1u);
          if (old == k) {
            rem[w] = tag;
            want = true;
          }
        }
      }
      push_warp(want, w, next, ncnt, cap, err);
    }
  }
}

// deg[v] = alive neighbours of v, for v in the alive list (big rows by blocks).
__global__ void k_recount(const uint32_t* __restrict__ alive, uint64_t n_alive, const uint64_t* __restrict__ off,
                          const uint32_t* __restrict__ adj, const uint32_t* __restrict__ rem,
                          uint32_t* __restrict__ deg, uint32_t* __restrict__ big, unsigned long long* nbig,
                          uint64_t cap, uint32_t* err, uint32_t big_row) {
  const uint64_t warps = (uint64_t)gridDim.x * (blockDim.x >> 5);
  for (uint64_t i = (uint64_t)blockIdx.x * (blockDim.x >> 5) + warp_id(); i < n_alive; i += warps) {
    const uint32_t v = alive[i];
    const uint64_t b = off[v], e = off[v + 1];
    if (e - b > big_row) {
      if (lane_id() == 0) {
        deg[v] = 0;
        const unsigned long long p = atomicAdd(nbig, 1ULL);
        if (p < cap)
          big[p] = v;
        else
          atomicOr(err, kDevErrCapacity);
      }
      continue;
    }
    uint32_t c = 0;
    for (uint64_t j = b + lane_id(); j < e; j += 32) c += rem[adj[j]] == kAlive;
    c = warp_sum(c);
    if (lane_id() == 0) deg[v] = c;
  }
}

// Big rows of the recount: their 256-entry windows dealt to every warp, 8
// entries per lane in flight, one atomic per window.
__global__ void __launch_bounds__(256) k_recount_big(const uint32_t* __restrict__ big,
                                                     const unsigned long long* nbig_p,
                                                     const uint64_t* __restrict__ off,
                                                     const uint32_t* __restrict__ adj,
                                                     const uint32_t* __restrict__ rem, uint32_t* __restrict__ deg) {
  __shared__ uint64_t woff[kBigBatch + 1];
  __shared__ uint64_t tmp[33];
  constexpr unsigned kPer = 8;
  deal_windows<32 * kPer>(
      *nbig_p, [&](uint64_t x) { return big[x]; }, off, woff, tmp, [&](uint64_t x, uint64_t b, uint64_t e) {
        const uint64_t j0 = b + lane_id();
        uint32_t w[kPer];
#pragma unroll
        for (unsigned k = 0; k < kPer; ++k) w[k] = j0 + 32 * k < e ? adj[j0 + 32 * k] : 0u;
        uint32_t n = 0;
#pragma unroll
        for (unsigned k = 0; k < kPer; ++k) n += j0 + 32 * k < e && rem[w[k]] == kAlive;
        n = warp_sum(n);
        if (lane_id() == 0 && n) atomicAdd(&deg[big[x]], n);
      });
}

__global__ void k_revive(uint32_t* __restrict__ rem, uint64_t n, uint32_t newer_than) {
  for (uint64_t v = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; v < n; v += (uint64_t)gridDim.x * blockDim.x) {
    const uint32_t r = rem[v];
    if (r != kAlive && r > newer_than) rem[v] = kAlive;
  }
}

// Minimum alive degree into *out; with `sum`, also the sum of the alive
// degrees (twice the alive edges).
__global__ void k_min_alive_deg(const uint32_t* __restrict__ alive, uint64_t n_alive, const uint32_t* __restrict__ deg,
                                const uint32_t* __restrict__ rem, uint32_t* out,
                                unsigned long long* sum = nullptr) {
  uint32_t mn = 0xffffffffu;
  uint64_t s = 0;
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n_alive; i += (uint64_t)gridDim.x * blockDim.x) {
    const uint32_t v = alive[i];
    if (rem[v] == kAlive) {
      mn = min(mn, deg[v]);
      s += deg[v];
    }
  }
  mn = warp_min(mn);
  if (lane_id() == 0 && mn != 0xffffffffu) atomicMin(out, mn);
  if (sum) {
    s = warp_sum(s);
    if (lane_id() == 0 && s) atomicAdd(sum, (unsigned long long)s);
  }
}

__global__ void k_members(const uint32_t* __restrict__ rem, uint64_t n, uint8_t* __restrict__ out) {
  for (uint64_t v = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; v < n; v += (uint64_t)gridDim.x * blockDim.x)
    out[v] = rem[v] == kAlive;
}

__global__ void k_core_from_tags(const uint32_t* __restrict__ rem, uint64_t n, const uint32_t* __restrict__ level,
                                 uint32_t* __restrict__ core) {
  for (uint64_t v = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; v < n; v += (uint64_t)gridDim.x * blockDim.x) {
    const uint32_t r = rem[v];
    core[v] = r == kAlive ? 0u : level[r] - 1;
  }
}


__global__ void k_compact_meta(const uint32_t* __restrict__ alive, uint64_t na, const uint32_t* __restrict__ deg,
                               const uint32_t* __restrict__ oldmap, uint32_t* __restrict__ newid,
                               uint32_t* __restrict__ ndeg, uint32_t* __restrict__ nmap) {
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < na; i += (uint64_t)gridDim.x * blockDim.x) {
    const uint32_t v = alive[i];
    newid[v] = (uint32_t)i;
    ndeg[i] = deg[v];
    nmap[i] = oldmap ? oldmap[v] : v;
  }
}

__global__ void k_members_mapped(const uint32_t* __restrict__ rem, uint64_t n, const uint32_t* __restrict__ map,
                                 uint8_t* __restrict__ out) {
  for (uint64_t v = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; v < n; v += (uint64_t)gridDim.x * blockDim.x)
    if (rem[v] == kAlive) out[map[v]] = 1;
}


// Rows of a frontier, 32 entries a step and kWide steps in flight, handed to
// `drop(w, ok)`: lane l of step t gets neighbour w[t] where ok[t].  A warp
// takes up to 32 vertices (fewer when the frontier is small for the grid) and
// walks their rows end to end, so short rows fill its lanes: a warp per vertex
// left most of them idle and waited for one entry after another (core
// decomposition of an R-MAT graph of 400,009 ids and 8M records: 5.3 -> 4.7 ms
// with this walk).  Rows longer than big_row go to big[0..*nbig).
constexpr unsigned kWide = 4;

template <class Drop>
__device__ __forceinline__ void walk_rows(const uint32_t* front, uint64_t nf,
                                          const uint64_t* __restrict__ off, const uint32_t* __restrict__ adj,
                                          uint32_t big_row, uint32_t* big, unsigned long long* nbig,
                                          uint64_t cap, uint32_t* err, Drop drop, Crew crew = Crew()) {
  const uint64_t gwarps = (uint64_t)crew.blocks * (blockDim.x >> 5);
  const uint64_t gwarp = (uint64_t)crew.rank * (blockDim.x >> 5) + warp_id();
  const unsigned lane = lane_id();
  const uint64_t share = (nf + gwarps - 1) / gwarps;
  const uint32_t per = share < 32 ? (uint32_t)share : 32u;
  for (uint64_t f0 = gwarp * per; f0 < nf; f0 += gwarps * per) {
    uint64_t start = 0;
    uint32_t len = 0, v = 0;
    if (lane < per && f0 + lane < nf) {
      v = front[f0 + lane];
      start = off[v];
      const uint64_t l = off[v + 1] - start;
      len = l > big_row ? 0xffffffffu : (uint32_t)l;
    }
    push_warp(len == 0xffffffffu, v, big, nbig, cap, err);
    if (len == 0xffffffffu) len = 0;
    const uint32_t incl = warp_incl_scan(len);
    const uint32_t total = __shfl_sync(kFull, incl, 31), excl = incl - len;
    start -= excl;  // entry p of the walk is adj[start + p] of its row's lane
    for (uint32_t base = 0; base < total; base += 32 * kWide) {
      uint32_t w[kWide];
      bool ok[kWide];
#pragma unroll
      for (unsigned t = 0; t < kWide; ++t) {
        const uint32_t p = base + 32 * t + lane;
        uint32_t from = 0;  // the last row starting at or before p
        if (per > 1) {
#pragma unroll
          for (uint32_t st = 16; st >= 1; st >>= 1) {
            const uint32_t x = __shfl_sync(kFull, excl, from + st);
            if (x <= p) from += st;
          }
        }
        const uint64_t s = __shfl_sync(kFull, start, from);
        ok[t] = p < total;
        w[t] = ok[t] ? adj[s + p] : 0u;
      }
      drop(w, ok);
    }
  }
}

// Threads of the cooperative kernels here, two blocks per SM: a barrier of 296
// blocks takes 1.6 us, of 592 blocks of 256 threads 2.3 (core decomposition of
// a 400,009-id R-MAT graph 4.94 -> 4.75 ms; one block of 1024 threads, which
// waits longer for its own warps, 5.10).
constexpr unsigned kCoreThreads = 512;

// What the search leaves for the host.
constexpr uint32_t kMaxProbes = 64;  // probes of one launch
struct SearchOut {
  uint64_t n_alive, rounds;
  uint32_t lo, hi;       // the lo-core is not empty, the hi-core is
  uint32_t ramp;         // still doubling
  uint32_t list;         // alive list in use (0 or 1)
  uint32_t probes;
  uint32_t compact;      // ended for a compaction (to the last probe's level)
  uint32_t k[kMaxProbes];
  uint32_t left[kMaxProbes];  // 0: the probe failed and was undone
};
static_assert(sizeof(SearchOut) <= 1024, "read through the context's pinned words");

struct SearchArgs {
  const uint64_t* off;
  const uint32_t* adj;
  uint32_t* deg;
  uint32_t* rem;
  uint32_t* snap;       // degrees before the probe, of the alive vertices (not fixed)
  uint32_t* alive[2];   // the list in use, and the one the next is written to
  uint64_t n_alive;
  // Frontier of the odd rounds; the even rounds' is the alive list not in use,
  // which the next list replaces once a probe's rounds are over.
  uint32_t* front;
  uint32_t* big;
  // [0..2] frontier sizes, [3..4] big-row counts, [5] least degree, [6] sum of
  // degrees; then one kept count per block
  unsigned long long* cnt;
  uint64_t cap;
  uint32_t lo, hi, ramp;  // search (lo, hi); hi = lo + 1 with fixed: one probe at level lo
  uint32_t fixed;
  uint32_t tag;           // of the first probe
  uint64_t compact_below; // end when the core's degrees add up to less than this
  uint32_t big_row;       // rows longer than this are dealt to all warps in windows
  SearchOut* out;
  DevWords* words;
  unsigned long long timeout_ns;
};

// Decrements the degrees of N neighbours per lane; the lanes' loads and
// atomics of all N are in flight before any result is used.
template <unsigned N>
__device__ __forceinline__ void drop_entries(const SearchArgs& A, const uint32_t (&w)[N], const bool (&ok)[N],
                                             uint32_t k, uint32_t tag, WarpList& next) {
  bool live[N];
#pragma unroll
  for (unsigned t = 0; t < N; ++t) live[t] = ok[t] && A.rem[w[t]] == kAlive;
  uint32_t old[N];
#pragma unroll
  for (unsigned t = 0; t < N; ++t) old[t] = live[t] ? atomicSub(&A.deg[w[t]], 1u) : 0u;
#pragma unroll
  for (unsigned t = 0; t < N; ++t) {
    const bool want = live[t] && old[t] == k;
    if (want) A.rem[w[t]] = tag;
    next.push(want, w[t]);
  }
}

// The maximum-core search in one cooperative launch.  Each probe starts with a
// pass over the alive list, which undoes a failed probe (degrees from the
// snapshot) or takes the snapshot, and picks the first frontier; then the
// rounds; a probe that leaves vertices ends with an ordered compaction of the
// alive list (each block counts and writes its own stretch of it) that also
// finds the least degree and the sum of the degrees.  With a launch per probe
// the host's reads and the launches between two probes cost 70 us of the 100
// us that a probe took on graphs of up to a million edges.
__global__ void __launch_bounds__(kCoreThreads, 2) k_core_search(SearchArgs A) {
  __shared__ uint32_t items[kCoreThreads / 32][WarpList::kEntries];
  __shared__ uint64_t woff[kBigBatch + 1];
  __shared__ uint64_t wtmp[33];
  __shared__ unsigned long long sh[2];
  const unsigned long long* src[2] = {nullptr, nullptr};
  const uint64_t gthreads = (uint64_t)gridDim.x * blockDim.x;
  const uint64_t gtid = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  unsigned long long* kept = A.cnt + 7;
  uint32_t lo = A.lo, hi = A.hi, ramp = A.ramp;
  uint64_t na = A.n_alive, rounds = 0;
  uint32_t list = 0, probes = 0, tag = A.tag, compact = 0;
  uint32_t i = 0;  // round index, continued across probes (it picks the counters)
  bool undo = false;
  auto front = [&](uint32_t round) { return (round & 1) ? A.front : A.alive[list ^ 1]; };
  while ((hi - lo > 1 || A.fixed) && na && probes < kMaxProbes) {
    uint32_t k;
    if (A.fixed) {
      k = lo;
    } else {
      k = ramp ? (2ull * lo < hi - 1 ? 2 * lo : hi - 1) : lo + (hi - lo) / 2;
      if (k <= lo) k = lo + 1;
    }
    // Slot (i + 1) % 3 is zero, and slot (i + 2) % 3 and the next round's big
    // count were read before the barriers of the rounds before.
    if (gtid == 0) {
      A.cnt[(i + 2) % 3] = 0;
      A.cnt[3 + ((i + 1) & 1)] = 0;
      A.cnt[5] = ~0ULL;
      A.cnt[6] = 0;
    }
    const uint32_t* alive = A.alive[list];
    WarpList first(items[warp_id()], front(i + 1), &A.cnt[(i + 1) % 3], A.cap, &A.words->err);
    for (uint64_t j = gtid; j < ((na + 31) & ~31ULL); j += gthreads) {
      bool want = false;
      uint32_t v = 0;
      if (j < na) {
        v = alive[j];
        uint32_t d;
        if (undo) {
          d = A.snap[v];
          A.deg[v] = d;
          A.rem[v] = kAlive;
        } else {
          d = A.deg[v];
          if (!A.fixed) A.snap[v] = d;
        }
        if (d < k) {
          A.rem[v] = tag;
          want = true;
        }
      }
      first.push(want, v);
    }
    first.flush();
    undo = false;
    ++i;
    src[0] = &A.cnt[i % 3];
    src[1] = nullptr;
    if (!grid_barrier_read(A.words, A.timeout_ns, src, sh)) return;
    uint64_t removed = 0;
    bool empty = false;
    while (true) {
      const uint64_t nf = sh[0];
      if (nf == 0) break;
      removed += nf;
      // Every block reads the same counts, so all of them stop together: fewer
      // than k+1 vertices can remain, so the k-core is empty.
      if (!A.fixed && na - removed < (uint64_t)k + 1) {
        empty = true;
        break;
      }
      const uint32_t* fr = front(i);
      unsigned long long* nc = &A.cnt[(i + 1) % 3];
      unsigned long long* bc = &A.cnt[3 + (i & 1)];
      WarpList next(items[warp_id()], front(i + 1), nc, A.cap, &A.words->err);
      walk_rows(
          fr, nf, A.off, A.adj, A.big_row, A.big, bc, A.cap, &A.words->err,
          [&](const uint32_t(&w)[kWide], const bool(&ok)[kWide]) { drop_entries<kWide>(A, w, ok, k, tag, next); });
      next.flush();
      if (gtid == 0) {
        A.cnt[(i + 2) % 3] = 0;        // read at the start of round i-1
        A.cnt[3 + ((i + 1) & 1)] = 0;  // big count of round i-1, read before the barrier ending it
      }
      // sh[0]: the next frontier's size so far (final when there are no big
      // rows, whose windows add to it); sh[1]: this round's big rows.
      src[0] = nc;
      src[1] = bc;
      if (!grid_barrier_read(A.words, A.timeout_ns, src, sh)) return;
      const uint64_t nbig = sh[1];
      if (nbig) {
        deal_windows<256>(
            nbig, [&](uint64_t x) { return A.big[x]; }, A.off, woff, wtmp, [&](uint64_t, uint64_t b, uint64_t e) {
              uint32_t w[8];
              bool ok[8];
#pragma unroll
              for (unsigned t = 0; t < 8; ++t) {
                const uint64_t j = b + lane_id() + 32 * t;
                ok[t] = j < e;
                w[t] = ok[t] ? A.adj[j] : 0u;
              }
              drop_entries<8>(A, w, ok, k, tag, next);
            });
        next.flush();
        if (!grid_barrier_read(A.words, A.timeout_ns, src, sh)) return;
      }
      ++i;
      ++rounds;
    }
    const uint64_t left = empty ? 0 : na - removed;
    if (gtid == 0) {
      A.out->k[probes] = k;
      A.out->left[probes] = (uint32_t)left;
    }
    ++probes;
    if (!left) {
      if (A.fixed) {
        na = 0;
        break;
      }
      hi = k;
      ramp = 0;
      undo = true;
      continue;
    }
    ++tag;
    // Ordered compaction: block b owns [b, b + 1) * stretch of the list.
    const uint64_t stretch = (na + gridDim.x - 1) / gridDim.x;
    const uint64_t s0 = min(na, blockIdx.x * stretch), s1 = min(na, s0 + stretch);
    uint64_t n = 0, sum = 0;
    uint32_t mn = 0xffffffffu;
    for (uint64_t j = s0 + threadIdx.x; j < s1; j += blockDim.x) {
      const uint32_t v = alive[j];
      if (A.rem[v] != kAlive) continue;
      const uint32_t d = A.deg[v];
      ++n;
      sum += d;
      mn = min(mn, d);
    }
    n = block_sum<uint64_t>(n, wtmp);
    mn = warp_min(mn);
    sum = warp_sum(sum);
    if (lane_id() == 0 && mn != 0xffffffffu) {
      atomicMin(&A.cnt[5], (unsigned long long)mn);
      atomicAdd(&A.cnt[6], (unsigned long long)sum);
    }
    if (threadIdx.x == 0) kept[blockIdx.x] = n;
    src[0] = &A.cnt[5];
    src[1] = &A.cnt[6];
    if (!grid_barrier_read(A.words, A.timeout_ns, src, sh)) return;
    const uint64_t dmin = sh[0], dsum = sh[1];
    uint64_t at = 0;
    for (uint32_t b = threadIdx.x; b < blockIdx.x; b += blockDim.x) at += ld_relaxed_u64(&kept[b]);
    at = block_sum<uint64_t>(at, wtmp);
    uint32_t* to = A.alive[list ^ 1];
    for (uint64_t j0 = s0; j0 < s1; j0 += blockDim.x) {
      const uint64_t j = j0 + threadIdx.x;
      const uint32_t v = j < s1 ? alive[j] : 0u;
      const bool keep = j < s1 && A.rem[v] == kAlive;
      uint64_t total;
      const uint64_t p = at + block_excl_scan<uint64_t>(keep ? 1 : 0, wtmp, &total);
      if (keep) to[p] = v;
      at += total;
    }
    list ^= 1;
    na = left;
    // The k-core left is the core of its least degree too, so every level up
    // to that is known to be non-empty.
    lo = k;
    if (dmin > lo) lo = dmin < hi - 1 ? (uint32_t)dmin : hi - 1;
    if (A.fixed) break;
    if (dsum < A.compact_below) {
      compact = 1;
      break;
    }
    if (!grid_barrier(A.words, A.timeout_ns)) return;
  }
  if (undo) {  // the last probe failed
    const uint32_t* alive = A.alive[list];
    for (uint64_t j = gtid; j < na; j += gthreads) {
      const uint32_t v = alive[j];
      A.deg[v] = A.snap[v];
      A.rem[v] = kAlive;
    }
  }
  if (gtid == 0) {
    SearchOut* o = A.out;
    o->n_alive = na;
    o->rounds = rounds;
    o->lo = lo;
    o->hi = hi;
    o->ramp = ramp;
    o->list = list;
    o->probes = probes;
    o->compact = compact;
  }
}

// Full core decomposition in one cooperative launch: the level loop runs on
// the device, so thousands of graphs of a batched union (or one graph) are
// decomposed without a host round trip per level.
//
// Level k removes every alive vertex of degree <= k (core number k): a pass
// over a vertex list takes the vertices of degree <= k as the first frontier,
// and the frontier rounds then run as in k_core_search (a neighbour stepping from
// k+1 to k joins the next frontier).  Passes are windowed: a full pass over
// the compact alive list opens a window of `window` levels [k, top] and
// lists the candidates, the alive vertices of degree <= top; within the
// window each level's pass reads only the candidates, and a neighbour whose
// degree steps from top+1 to top during the rounds joins them.  So the alive
// list is read once per window instead of once per level.  A pass that finds
// no vertex of degree k moves k to the smallest degree it saw (levels
// without vertices are skipped).
//
// The graphs of a union are decomposed by teams of blocks, each with a stretch
// of the graphs, a barrier and counters of its own: in step with each other,
// 64 graphs took 3,771 rounds where none of them alone takes more than 966, and
// a round is bound by the latency of its chain of accesses (33.5 ms, 9.4 by 28
// teams with 964 rounds at most).
struct Team {
  uint32_t block0, blocks;
  uint64_t v0, v1;     // its vertices
  uint64_t list0;      // its first entry of the alive list
  uint64_t n_list;
};
constexpr unsigned kMaxTeams = 64;
constexpr unsigned kTeamCounters = 24;
constexpr uint64_t kTeamEntries = 1u << 20;  // (the waves of small requests are no faster by teams)

struct DecompArgs {
  const Team* teams;   // nteams of them, or null: one of the whole grid
  uint32_t nteams;
  DevWords* team_words;
  const uint64_t* off;
  const uint32_t* adj;
  uint32_t* deg;
  uint32_t* rem;       // kAlive, or 0 once removed
  uint32_t* core;      // out: core number of every removed vertex
  uint32_t* list[2];   // compact alive lists (ping-pong, rewritten by full passes)
  uint32_t* cand[2];   // window candidates (ping-pong, rewritten by every pass)
  uint32_t* front[2];
  uint32_t* big;
  // [0..2] frontier sizes, [3..4] big-row counts; by pass % 3: [5..7]
  // alive-list sizes, [8..10] minimum degrees, [11..13] candidate counts;
  // [14] rounds, [15] levels, [16] passes, [17] full passes, [18] last level
  unsigned long long* cnt;
  uint64_t n_list;     // entries of list[0] at launch
  uint64_t cap;
  uint32_t big_row;    // rows longer than this are dealt to all warps in windows
  uint32_t window;     // levels per window (>= 1)
  DevWords* words;
  unsigned long long timeout_ns;
};

template <unsigned N>
__device__ __forceinline__ void drop_entries_core(const DecompArgs& A, const uint32_t (&w)[N], const bool (&ok)[N],
                                                  uint32_t k, uint32_t top, WarpList& next, WarpList& cand) {
  bool live[N];
#pragma unroll
  for (unsigned t = 0; t < N; ++t) live[t] = ok[t] && A.rem[w[t]] == kAlive;
  uint32_t old[N];
#pragma unroll
  for (unsigned t = 0; t < N; ++t) old[t] = live[t] ? atomicSub(&A.deg[w[t]], 1u) : 0u;
#pragma unroll
  for (unsigned t = 0; t < N; ++t) {
    const bool want = live[t] && old[t] == k + 1;
    const bool join = live[t] && !want && old[t] == top + 1;  // its degree entered the window
    if (want) {
      A.rem[w[t]] = 0u;
      A.core[w[t]] = k;
    }
    next.push(want, w[t]);
    cand.push(join, w[t]);
  }
}

// The entries of the alive list in each team's vertices, and its least degrees
// at their start.
__global__ void k_team_lists(Team* __restrict__ teams, uint32_t nteams, const uint32_t* __restrict__ alive,
                             uint64_t n_alive, unsigned long long* __restrict__ cnt) {
  const uint32_t t = threadIdx.x;
  if (t >= nteams) return;
  for (int q = 8; q < 11; ++q) cnt[t * kTeamCounters + q] = ~0ULL;
  uint64_t at[2];
  for (int q = 0; q < 2; ++q) {
    const uint64_t v = q ? teams[t].v1 : teams[t].v0;
    uint64_t lo = 0, hi = n_alive;
    while (lo < hi) {
      const uint64_t mid = (lo + hi) >> 1;
      if (alive[mid] < v)
        lo = mid + 1;
      else
        hi = mid;
    }
    at[q] = lo;
  }
  teams[t].list0 = at[0];
  teams[t].n_list = at[1] - at[0];
}

template <bool kTeams>
__global__ void __launch_bounds__(kCoreThreads, 2) k_core_levels(const __grid_constant__ DecompArgs args) {
  __shared__ DecompArgs mine;
  __shared__ unsigned team_block0, team_blocks;
  if (kTeams && threadIdx.x == 0) {
    uint32_t t = 0;
    while (t + 1 < args.nteams && args.teams[t + 1].block0 <= blockIdx.x) ++t;
    const Team T = args.teams[t];
    team_block0 = T.block0;
    team_blocks = T.blocks;
    mine = args;
    // Each list's stretch of the team holds as many entries as it has vertices.
    mine.list[0] += T.list0;
    mine.list[1] += T.v0;
    for (int q = 0; q < 2; ++q) {
      mine.cand[q] += T.v0;
      mine.front[q] += T.v0;
    }
    mine.big += T.v0;
    mine.cnt += kTeamCounters * t;
    mine.n_list = T.n_list;
    mine.cap = T.v1 - T.v0;
    mine.words = args.team_words + t;
  }
  __syncthreads();
  const DecompArgs& A = kTeams ? mine : args;
  const Crew crew = kTeams ? Crew(blockIdx.x - team_block0, team_blocks) : Crew();
  __shared__ unsigned long long sh[4];
  __shared__ uint32_t items[3][kCoreThreads / 32][WarpList::kEntries];
  __shared__ uint64_t woff[kBigBatch + 1];
  __shared__ uint64_t wtmp[33];
  const uint64_t gthreads = (uint64_t)crew.blocks * blockDim.x;
  const uint64_t gtid = (uint64_t)crew.rank * blockDim.x + threadIdx.x;
  uint64_t nl = A.n_list;  // entries of the current alive list
  uint64_t nc = 0;         // entries of the current candidate list
  uint32_t k = 1;          // every alive vertex has degree >= k
  uint32_t top = 0;        // candidates: every alive vertex of degree <= top
  bool full = true;        // the next pass reads the alive list
  uint32_t i = 0;          // frontier round index, continued across levels
  uint32_t ps = 0, li = 0, ci = 0;
  unsigned long long levels_run = 0, full_passes = 0;
  while (true) {
    unsigned long long* lc = &A.cnt[5 + ps % 3];
    unsigned long long* mc = &A.cnt[8 + ps % 3];
    unsigned long long* cc = &A.cnt[11 + ps % 3];
    if (gtid == 0) {
      // Read two passes ago, before the barriers that ended the last pass.
      A.cnt[5 + (ps + 1) % 3] = 0;
      A.cnt[8 + (ps + 1) % 3] = ~0ULL;
      A.cnt[11 + (ps + 1) % 3] = 0;
      // The pass pushes the frontier of round i + 1.  Slot i % 3 (empty; it
      // ended the last level) may still be being read by slower blocks, so it
      // is left alone; slot (i + 2) % 3 and round i + 1's big-row count were
      // read before the barriers that ended round i - 1, and are cleared.
      A.cnt[(i + 2) % 3] = 0;
      A.cnt[3 + ((i + 1) & 1)] = 0;
    }
    if (full) {
      top = k + A.window - 1;
      ++full_passes;
    }
    const uint32_t* src = full ? (li ? A.list[1] : A.list[0]) : (ci ? A.cand[1] : A.cand[0]);
    const uint64_t nsrc = full ? nl : nc;
    uint32_t* lnext = li ? A.list[0] : A.list[1];
    uint32_t* cnext = ci ? A.cand[0] : A.cand[1];
    uint32_t mn = 0xffffffffu;
    WarpList cands(items[1][warp_id()], cnext, cc, A.cap, &A.words->err);
    WarpList leaving(items[0][warp_id()], (i & 1) ? A.front[0] : A.front[1], &A.cnt[(i + 1) % 3], A.cap,
                     &A.words->err);
    WarpList staying(items[2][warp_id()], lnext, lc, A.cap, &A.words->err);
    for (uint64_t j = gtid; j < ((nsrc + 31) & ~31ULL); j += gthreads) {
      bool out = false, keep = false, cand = false;
      uint32_t v = 0;
      if (j < nsrc) {
        v = src[j];
        if (A.rem[v] == kAlive) {
          const uint32_t d = A.deg[v];
          if (d <= k) {
            A.rem[v] = 0u;
            A.core[v] = k;
            out = true;
          } else {
            keep = full;
            cand = d <= top;
            mn = min(mn, d);
          }
        }
      }
      leaving.push(out, v);
      if (full) staying.push(keep, v);
      cands.push(cand, v);
    }
    leaving.flush();
    staying.flush();
    cands.flush();
    mn = warp_min(mn);
    if (lane_id() == 0 && mn != 0xffffffffu) atomicMin(mc, (unsigned long long)mn);
    {
      const unsigned long long* const src[4] = {lc, mc, cc, &A.cnt[(i + 1) % 3]};
      if (!grid_barrier_read(A.words, A.timeout_ns, src, sh, crew)) return;
    }
    if (full) {
      nl = sh[0];
      li ^= 1;
    }
    const unsigned long long dmin = sh[1];
    uint64_t nf = sh[3];
    ++ps;
    // The pass's frontier is round i + 1's; i advances even when it is empty,
    // so the next pass counts into a slot no slower block is still reading.
    ++i;
    if (nf == 0) {
      nc = sh[2];
      ci ^= 1;
      if (full) {
        if (nl == 0) break;  // nothing alive
        k = (uint32_t)dmin;  // the candidates hold level dmin's vertices when it is in the window
        full = k > top;
      } else if (nc) {
        k = (uint32_t)dmin;  // the smallest candidate degree (<= top)
      } else {
        k = top + 1;  // no alive vertex of degree <= top: open the next window
        full = true;
      }
      continue;
    }
    ++levels_run;
    // Frontier rounds of level k.
    while (nf) {
      const uint32_t* fr = (i & 1) ? A.front[1] : A.front[0];
      WarpList next(items[0][warp_id()], (i & 1) ? A.front[0] : A.front[1], &A.cnt[(i + 1) % 3], A.cap,
                    &A.words->err);
      unsigned long long* bc = &A.cnt[3 + (i & 1)];
      walk_rows(fr, nf, A.off, A.adj, A.big_row, A.big, bc, A.cap, &A.words->err,
                [&](const uint32_t(&w)[kWide], const bool(&ok)[kWide]) {
                  drop_entries_core<kWide>(A, w, ok, k, top, next, cands);
                },
                crew);
      next.flush();
      cands.flush();
      if (gtid == 0) {
        A.cnt[(i + 2) % 3] = 0;
        A.cnt[3 + ((i + 1) & 1)] = 0;
      }
      const unsigned long long* const src[3] = {next.cnt, bc, cc};
      if (!grid_barrier_read(A.words, A.timeout_ns, src, sh, crew)) return;
      const uint64_t nbig = sh[1];
      if (nbig) {
        deal_windows<128>(
            nbig, [&](uint64_t x) { return A.big[x]; }, A.off, woff, wtmp, [&](uint64_t, uint64_t b, uint64_t e) {
              uint32_t w[4];
              bool ok[4];
#pragma unroll
              for (unsigned t = 0; t < 4; ++t) {
                const uint64_t j = b + lane_id() + 32 * t;
                ok[t] = j < e;
                w[t] = ok[t] ? A.adj[j] : 0u;
              }
              drop_entries_core<4>(A, w, ok, k, top, next, cands);
            },
            crew);
        next.flush();
        cands.flush();
        if (!grid_barrier_read(A.words, A.timeout_ns, src, sh, crew)) return;
      }
      nf = sh[0];
      ++i;
    }
    // Every candidate push of this pass is in (rounds end with a barrier).
    nc = sh[2];
    ci ^= 1;
    ++k;  // every survivor now has degree >= k
    full = k > top;
  }
  if (gtid == 0) {
    A.cnt[14] = i;
    A.cnt[15] = levels_run;
    A.cnt[16] = ps;
    A.cnt[17] = full_passes;
    A.cnt[18] = k;
  }
}

// Blocks of a cooperative launch here at most (one count per block is kept).
constexpr unsigned kMaxGrid = 4096;
// Graphs with fewer edges (32 MB of adjacency) are searched without compaction:
// the copy cost more than the probes it sped up (R-MAT scale 18, 3.4M edges:
// membership of one core 1.26 ms with copies, 1.09 ms without; a 49M-edge
// Chung-Lu solve 21.8 ms with, 22.3 ms without).
constexpr uint64_t kCompactMinEdges = 1u << 22;

uint32_t big_row(const Ctx* c) {
  // At most 2^26: a warp adds up the lengths of 32 rows in 32 bits.
  return (uint32_t)std::min<int64_t>(std::max<int64_t>(32, c->opt.kcore_big_row), 1 << 26);
}

}  // namespace

void KCore::ensure_state(Ctx* c, const Graph& gr) {
  n = gr.n;
  deg.ensure(c, (n ? n : 1) * sizeof(uint32_t));
  rem.ensure(c, (n ? n : 1) * sizeof(uint32_t));
  alive.ensure(c, (n ? n : 1) * sizeof(uint32_t));
  front[0].ensure(c, (n ? n : 1) * sizeof(uint32_t));
  front[1].ensure(c, (n ? n : 1) * sizeof(uint32_t));
  big.ensure(c, (n ? n : 1) * sizeof(uint32_t));
  cnt.ensure(c, (7 + kMaxGrid) * sizeof(unsigned long long));
}

void KCore::reset_state(Ctx* c, const Graph& gr) {
  ensure_state(c, gr);
  if (n) {
    k_init_state<<<grid_for(n, 256, c->num_sms * 16), 256, 0, c->stream>>>(gr.deg.as<uint32_t>(), n,
                                                                             deg.as<uint32_t>(), rem.as<uint32_t>());
    KT_LAUNCHED(c);
  }
  rebuild_alive(c);
}

void KCore::init(Ctx* c, const Graph& gr) {
  base = &gr;
  saved.clear();
  compacted = false;
  local_level = 0;
  levels.assign(1, 1);  // tag 0 = isolated, left at level 1
  succ.assign(1, 0);
  reset_state(c, gr);
}

void KCore::rebuild_alive(Ctx* c) {
  n_alive = compact(c, n, AliveF{rem.as<uint32_t>()}, alive.as<uint32_t>());
}

void KCore::compact_to_alive(Ctx* c, uint32_t level) {
  const Graph& g = cur();
  const uint64_t na = n_alive;
  Graph L;
  L.n = na;
  DBuf newid(c, (n ? n : 1) * sizeof(uint32_t));
  DBuf nmap(c, (na ? na : 1) * sizeof(uint32_t));
  L.deg.alloc(c, (na + 1) * sizeof(uint32_t));
  zero(c, L.deg.get(), (na + 1) * sizeof(uint32_t));
  k_compact_meta<<<grid_for(na, 256, c->num_sms * 16), 256, 0, c->stream>>>(
      alive.as<uint32_t>(), na, deg.as<uint32_t>(), map(), newid.as<uint32_t>(), L.deg.as<uint32_t>(),
      nmap.as<uint32_t>());
  KT_LAUNCHED(c);
  L.off.alloc(c, (na + 1) * sizeof(uint64_t));
  scan_u32_to_u64(c, L.deg.as<uint32_t>(), L.off.as<uint64_t>(), na + 1);
  const uint64_t n2 = read_word<uint64_t>(c, L.off.as<uint64_t>() + na);
  L.m = n2 / 2;
  L.adj.alloc(c, (n2 ? n2 : 1) * sizeof(uint32_t));
  copy_rows(c, alive.as<uint32_t>(), na, g.off.as<uint64_t>(), g.adj.as<uint32_t>(), rem.as<uint32_t>(),
            newid.as<uint32_t>(), L.off.as<uint64_t>(), g.max_deg, OutColumn{L.adj.as<uint32_t>()});
  L.max_deg = g.max_deg;  // an upper bound is enough here
  newid.release();
  // Install; what was worked on so far is kept for restores.  (Its tags stay in
  // their buffer; the ones freed here make up for that.)
  Saved sv;
  sv.rem = std::move(rem);
  sv.levels = std::move(levels);
  sv.succ = std::move(succ);
  if (compacted) {
    sv.local = std::move(local);
    sv.idmap = std::move(idmap);
    sv.level = local_level;
    local = Graph();
  }
  saved.push_back(std::move(sv));
  rem = std::move(snap);
  front[0].release();
  front[1].release();
  big.release();
  local.off = std::move(L.off);
  local.adj = std::move(L.adj);
  local.deg = std::move(L.deg);
  local.edges.release();
  local.n = L.n;
  local.m = L.m;
  local.max_deg = L.max_deg;
  idmap = std::move(nmap);
  compacted = true;
  local_level = level;
  levels.assign(1, level);
  succ.assign(1, 0);
  reset_state(c, local);
}

void KCore::recount(Ctx* c) {
  if (!n_alive) return;
  const Graph& g = cur();
  zero(c, cnt.get(), cnt.bytes());
  unsigned long long* nbig = cnt.as<unsigned long long>() + 4;
  k_recount<<<grid_for(n_alive * 32, 256, c->num_sms * 16), 256, 0, c->stream>>>(
      alive.as<uint32_t>(), n_alive, g.off.as<uint64_t>(), g.adj.as<uint32_t>(), rem.as<uint32_t>(),
      deg.as<uint32_t>(), big.as<uint32_t>(), nbig, n, &dev_words(c)->err, big_row(c));
  KT_LAUNCHED(c);
  k_recount_big<<<c->num_sms * 8, 256, 0, c->stream>>>(big.as<uint32_t>(), nbig, g.off.as<uint64_t>(),
                                                       g.adj.as<uint32_t>(), rem.as<uint32_t>(),
                                                       deg.as<uint32_t>());
  KT_LAUNCHED(c);
}

// One launch of k_core_search from the current alive set: the search of
// (lo, hi), or with fixed one probe at level lo.  Successful probes get their
// tags, and the alive list and n_alive are the last one's.
void KCore::search_launch(Ctx* c, uint32_t lo, uint32_t hi, bool ramp, bool fixed, uint64_t compact_below,
                          void* result) {
  const Graph& g = cur();
  if (!fixed) snap.ensure(c, (n ? n : 1) * sizeof(uint32_t));
  out.ensure(c, sizeof(SearchOut));
  if (!coop_grid) {
    int per_sm = 0;
    KT_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_core_search, kCoreThreads, 0));
    coop_grid = std::min(coop_blocks(c, per_sm), kMaxGrid);
  }
  SearchArgs A;
  A.off = g.off.as<uint64_t>();
  A.adj = g.adj.as<uint32_t>();
  A.deg = deg.as<uint32_t>();
  A.rem = rem.as<uint32_t>();
  A.snap = snap.as<uint32_t>();
  A.alive[0] = alive.as<uint32_t>();
  A.alive[1] = front[0].as<uint32_t>();
  A.n_alive = n_alive;
  A.front = front[1].as<uint32_t>();
  A.big = big.as<uint32_t>();
  A.cnt = cnt.as<unsigned long long>();
  A.cap = n;
  A.lo = lo;
  A.hi = hi;
  A.ramp = ramp;
  A.fixed = fixed;
  A.tag = (uint32_t)levels.size();
  A.compact_below = compact_below;
  A.big_row = big_row(c);
  A.out = out.as<SearchOut>();
  A.words = dev_words(c);
  A.timeout_ns = (unsigned long long)c->opt.timeout_ms * 1000000ULL;
  if (A.tag >= 0xfffffff0u - kMaxProbes) throw Error(KT_ERR_LIMIT, "k-core: too many probes");
  zero(c, cnt.get(), 7 * sizeof(unsigned long long));
  void* p[] = {&A};
  SearchOut& h = *static_cast<SearchOut*>(result);
  {
    CoopLock coop(c);
    const unsigned grid = coop_blocks_for(coop_grid, 2 * g.m, kCoreThreads * kWide);
    KT_CUDA(cudaLaunchCooperativeKernel((const void*)k_core_search, dim3(grid), dim3(kCoreThreads), p, 0, c->stream));
    KT_LAUNCHED(c);
    read_checked(c, &h, out.get(), sizeof(SearchOut), "k-core probe");
  }
  rounds += h.rounds;
  probes += h.probes;
  n_alive = h.n_alive;
  if (h.list) std::swap(alive, front[0]);
  for (uint32_t i = 0; i < h.probes; ++i) {
    KT_LOG(c, "kt: k-core probe %u: %u vertices left\n", h.k[i], h.left[i]);
    if (!h.left[i] && !fixed) continue;
    if (!fixed) succ.push_back((uint32_t)levels.size());
    levels.push_back(h.k[i]);
  }
}

uint64_t KCore::probe(Ctx* c, uint32_t k, bool may_stop) {
  if (!n_alive) {
    levels.push_back(k);
    return 0;
  }
  if (c->opt.persistent) {
    SearchOut h;
    search_launch(c, k, k + 1, false, true, 0, &h);
    return n_alive;
  }
  const uint32_t tag = (uint32_t)levels.size();
  if (tag >= 0xfffffff0u) throw Error(KT_ERR_LIMIT, "k-core: too many probes");
  levels.push_back(k);
  const Graph& g = cur();
  unsigned long long* cn = cnt.as<unsigned long long>();
  zero(c, cnt.get(), 7 * sizeof(unsigned long long));
  uint32_t* err = &dev_words(c)->err;
  uint64_t removed = 0;
  {
    k_frontier_init<<<grid_for(n_alive, 256, c->num_sms * 16), 256, 0, c->stream>>>(
        alive.as<uint32_t>(), n_alive, deg.as<uint32_t>(), rem.as<uint32_t>(), k, tag, front[0].as<uint32_t>(),
        cn + 0, n, err);
    KT_LAUNCHED(c);
    int cur_f = 0;
    while (true) {
      const uint64_t nf = read_word<unsigned long long>(c, cn + cur_f);
      if (nf == 0) break;
      removed += nf;
      if (may_stop && n_alive - removed < (uint64_t)k + 1) {
        removed = n_alive;  // the k-core is empty (the state is partial)
        break;
      }
      ++rounds;
      KT_CUDA(cudaMemsetAsync(cn + (cur_f ^ 1), 0, sizeof(unsigned long long), c->stream));
      KT_CUDA(cudaMemsetAsync(cn + 4, 0, sizeof(unsigned long long), c->stream));
      k_expand<<<grid_for(nf * 32, 256, c->num_sms * 16), 256, 0, c->stream>>>(
          front[cur_f].as<uint32_t>(), nf, g.off.as<uint64_t>(), g.adj.as<uint32_t>(), deg.as<uint32_t>(),
          rem.as<uint32_t>(), k, tag, front[cur_f ^ 1].as<uint32_t>(), cn + (cur_f ^ 1), big.as<uint32_t>(),
          cn + 4, n, err, big_row(c));
      KT_LAUNCHED(c);
      k_expand_big<<<c->num_sms * 4, 256, 0, c->stream>>>(big.as<uint32_t>(), cn + 4, g.off.as<uint64_t>(),
                                                          g.adj.as<uint32_t>(), deg.as<uint32_t>(),
                                                          rem.as<uint32_t>(), k, tag, front[cur_f ^ 1].as<uint32_t>(),
                                                          cn + (cur_f ^ 1), n, err);
      KT_LAUNCHED(c);
      cur_f ^= 1;
    }
  }
  ++probes;
  check_words(c, "k-core probe");
  const uint64_t left = n_alive - removed;
  if (left) rebuild_alive(c);
  return left;
}

uint32_t KCore::find_max_core(Ctx* c) {
  if (!n_alive) {
    cmax = 0;
    return 0;
  }
  // Upper bound: a k-core holds >= k(k+1)/2 edges.
  const double m = (double)base->m;
  uint64_t ub = (uint64_t)std::floor((std::sqrt(1.0 + 8.0 * m) - 1.0) / 2.0);
  ub = std::min<uint64_t>(ub, base->max_deg);
  uint64_t lo = 1, hi = ub + 1;  // the 1-core (non-isolated vertices) is non-empty
  bool ramp = true;
  if (c->opt.persistent) {
    while (hi - lo > 1) {
      // Work on a compacted copy once the core's edges are a small part of
      // the current graph's: a copy that keeps most of them costs more than
      // the probes it would speed up.  (The copy holds the k-core, which
      // every level from k up can be restored from.)  A graph below
      // kCompactMinEdges stays as it is: it is read from L2 either way.
      const uint64_t m2 = 2 * cur().m;
      const uint64_t below = c->opt.kcore_compact > 0 && cur().m >= kCompactMinEdges
                                 ? (m2 + c->opt.kcore_compact - 1) / (uint64_t)c->opt.kcore_compact
                                 : 0;
      SearchOut h;
      search_launch(c, (uint32_t)lo, (uint32_t)hi, ramp, false, below, &h);
      lo = h.lo;
      hi = h.hi;
      ramp = h.ramp;
      if (h.compact) {
        const uint32_t k = h.k[h.probes - 1];
        compact_to_alive(c, k);
        KT_LOG(c, "kt: k-core compacted copy of the %u-core: %llu vertices, %llu edges\n", k,
               (unsigned long long)n, (unsigned long long)local.m);
      }
    }
    snap.release();
    cmax = (uint32_t)lo;
    return cmax;
  }
  DBuf mn(c, 16), snap;
  while (hi - lo > 1) {
    uint64_t k = ramp ? std::min<uint64_t>(lo * 2, hi - 1) : lo + (hi - lo) / 2;
    if (k <= lo) k = lo + 1;
    const uint32_t tag = (uint32_t)levels.size();
    const auto t0 = std::chrono::steady_clock::now();
    const uint64_t before = n_alive;
    // Degrees before the probe: a failed probe is undone by reviving its tag
    // and copying them back (the alive set is then the one they belong to).
    snap.ensure(c, n * sizeof(uint32_t));
    KT_CUDA(cudaMemcpyAsync(snap.get(), deg.get(), n * sizeof(uint32_t), cudaMemcpyDeviceToDevice, c->stream));
    const uint64_t left = probe(c, (uint32_t)k, true);
    KT_LOG(c, "kt: k-core probe %llu: %llu of %llu alive vertices left, %.3f ms\n", (unsigned long long)k,
           (unsigned long long)left, (unsigned long long)before,
           std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now() - t0).count());
    if (left) {
      lo = k;
      succ.push_back(tag);
      // The probe left the k-core; its minimum degree d >= k makes it the
      // d-core too, so every level up to d is known to be non-empty.
      // mn: [0] the minimum alive degree, [2..3] the sum of alive degrees.
      KT_CUDA(cudaMemsetAsync(mn.get(), 0xff, 4, c->stream));
      KT_CUDA(cudaMemsetAsync(mn.as<uint32_t>() + 2, 0, 8, c->stream));
      k_min_alive_deg<<<grid_for(n_alive, 256, c->num_sms * 8), 256, 0, c->stream>>>(
          alive.as<uint32_t>(), n_alive, deg.as<uint32_t>(), rem.as<uint32_t>(), mn.as<uint32_t>(),
          reinterpret_cast<unsigned long long*>(mn.as<uint32_t>() + 2));
      KT_LAUNCHED(c);
      uint32_t h[4];
      copy_d2h(c, h, mn.get(), sizeof(h));
      const uint32_t d = h[0];
      uint64_t deg_sum = 0;
      std::memcpy(&deg_sum, h + 2, 8);
      if (d != 0xffffffffu && d > lo) lo = std::min<uint64_t>(d, hi - 1);
      // Work on a compacted copy once the core's edges are a small part of
      // the current graph's: a copy that keeps most of them costs more than
      // the probes it would speed up.  (The copy holds the k-core, which
      // every level from k up can be restored from.)
      if (c->opt.kcore_compact > 0 && (deg_sum / 2) * (uint64_t)c->opt.kcore_compact < cur().m) {
        const auto tc = std::chrono::steady_clock::now();
        const uint64_t from = n;
        compact_to_alive(c, (uint32_t)k);
        KT_LOG(c, "kt: k-core compacted copy of the %llu-core: %llu of %llu vertices, %llu edges, %.3f ms\n",
               (unsigned long long)k, (unsigned long long)n, (unsigned long long)from,
               (unsigned long long)local.m,
               std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now() - tc).count());
      }
    } else {
      hi = k;
      ramp = false;
      // Undo: revive this probe's vertices and restore their degrees.
      k_revive<<<grid_for(n, 256, c->num_sms * 16), 256, 0, c->stream>>>(rem.as<uint32_t>(), n, tag - 1);
      KT_LAUNCHED(c);
      levels.pop_back();
      KT_CUDA(cudaMemcpyAsync(deg.get(), snap.get(), n * sizeof(uint32_t), cudaMemcpyDeviceToDevice, c->stream));
    }
  }
  cmax = (uint32_t)lo;
  return cmax;
}

void KCore::restore_core(Ctx* c, uint32_t k) {
  if (compacted && k < local_level) {
    // Below the compacted core: back to the deepest earlier graph whose level
    // is at or below k, the input graph at the least.
    while (saved.back().level > k) saved.pop_back();
    Saved& sv = saved.back();
    compacted = sv.level != 0;
    local = std::move(sv.local);
    idmap = std::move(sv.idmap);
    local_level = sv.level;
    rem = std::move(sv.rem);
    levels = std::move(sv.levels);
    succ = std::move(sv.succ);
    saved.pop_back();
    ensure_state(c, cur());
  }
  // Last successful probe at or below level k; everything newer is revived.
  uint32_t keep = 0;
  for (uint32_t t : succ)
    if (levels[t] <= k) keep = std::max(keep, t);
  levels.resize(keep + 1);
  std::vector<uint32_t> s2;
  for (uint32_t t : succ)
    if (t <= keep) s2.push_back(t);
  succ.swap(s2);
  if (keep == 0) {
    reset_state(c, cur());  // every vertex with edges, at the graph's own degrees
  } else {
    k_revive<<<grid_for(n, 256, c->num_sms * 16), 256, 0, c->stream>>>(rem.as<uint32_t>(), n, keep);
    KT_LAUNCHED(c);
    rebuild_alive(c);
    recount(c);
  }
  const uint32_t tag = (uint32_t)levels.size();
  if (probe(c, k)) succ.push_back(tag);
}

void KCore::members(Ctx* c, uint8_t* dout) {
  if (!base->n) return;
  if (compacted) {
    zero(c, dout, base->n);
    if (n) {
      k_members_mapped<<<grid_for(n, 256, c->num_sms * 16), 256, 0, c->stream>>>(rem.as<uint32_t>(), n,
                                                                                   idmap.as<uint32_t>(), dout);
      KT_LAUNCHED(c);
    }
    return;
  }
  k_members<<<grid_for(n, 256, c->num_sms * 16), 256, 0, c->stream>>>(rem.as<uint32_t>(), n, dout);
  KT_LAUNCHED(c);
}

void KCore::core_numbers(Ctx* c, uint32_t* dcore, const std::vector<uint64_t>* starts) {
  if (compacted) throw Error(KT_ERR_INVALID, "core_numbers needs an uncompacted state");
  if (c->opt.persistent) {
    core_numbers_persistent(c, dcore, starts);
    return;
  }
  // Peel level by level: the alive set is always a d-core where d is its
  // minimum degree, so the probe at d+1 removes exactly the core-d vertices.
  DBuf mn(c, 4);
  while (n_alive) {
    KT_CUDA(cudaMemsetAsync(mn.get(), 0xff, 4, c->stream));
    k_min_alive_deg<<<grid_for(n_alive, 256, c->num_sms * 8), 256, 0, c->stream>>>(
        alive.as<uint32_t>(), n_alive, deg.as<uint32_t>(), rem.as<uint32_t>(), mn.as<uint32_t>());
    KT_LAUNCHED(c);
    const uint32_t d = read_word<uint32_t>(c, mn.as<uint32_t>());
    n_alive = probe(c, d + 1);
  }
  DBuf lv(c, levels.size() * sizeof(uint32_t));
  copy_h2d(c, lv.get(), levels.data(), levels.size() * sizeof(uint32_t));
  if (n) {
    k_core_from_tags<<<grid_for(n, 256, c->num_sms * 16), 256, 0, c->stream>>>(rem.as<uint32_t>(), n,
                                                                                 lv.as<uint32_t>(), dcore);
    KT_LAUNCHED(c);
  }
  sync(c);
}

}  // namespace kt

namespace kt {

// Teams of a union's graphs (vertices starts[g] .. starts[g + 1]) by edges.
static std::vector<Team> make_teams(Ctx* c, const Graph& g, const std::vector<uint64_t>& starts, unsigned grid) {
  std::vector<Team> teams;
  if (starts.size() < 3 || 2 * g.m < kTeamEntries) return teams;
  for (const TeamSpan& t : split_teams(gather_offsets(c, g.off.as<uint64_t>(), starts), kMaxTeams, grid))
    teams.push_back(Team{t.block0, t.blocks, starts[t.first], starts[t.last], 0, 0});
  return teams;
}

void KCore::core_numbers_persistent(Ctx* c, uint32_t* dcore, const std::vector<uint64_t>* starts) {
  if (!n) return;
  zero(c, dcore, n * sizeof(uint32_t));  // isolated vertices: core 0
  if (!n_alive) return;
  const Graph& g = cur();
  DBuf list2(c, n * sizeof(uint32_t)), cand0(c, n * sizeof(uint32_t)), cand1(c, n * sizeof(uint32_t));
  int per_sm = 0;
  KT_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_core_levels<true>, kCoreThreads, 0));
  if (c->opt.kcore_blocks_per_sm > 0) per_sm = (int)std::min<int64_t>(per_sm, c->opt.kcore_blocks_per_sm);
  unsigned grid = coop_blocks_for(coop_blocks(c, per_sm), 2 * g.m, kCoreThreads * kWide);
  std::vector<Team> teams;
  if (starts) teams = make_teams(c, g, *starts, grid);
  const unsigned nteams = std::max<unsigned>(1, (unsigned)teams.size());
  DBuf cn(c, nteams * kTeamCounters * sizeof(unsigned long long));
  zero(c, cn.get(), cn.bytes());
  DBuf dteams, words;
  if (!teams.empty()) {
    grid = teams.back().block0 + teams.back().blocks;
    dteams.alloc(c, teams.size() * sizeof(Team));
    copy_h2d(c, dteams.get(), teams.data(), teams.size() * sizeof(Team));
    words.alloc(c, teams.size() * sizeof(DevWords));
    zero(c, words.get(), words.bytes());
    k_team_lists<<<1, kMaxTeams, 0, c->stream>>>(dteams.as<Team>(), nteams, alive.as<uint32_t>(), n_alive,
                                                 cn.as<unsigned long long>());
    KT_LAUNCHED(c);
  } else {
    KT_CUDA(cudaMemsetAsync(cn.as<unsigned long long>() + 8, 0xff, 3 * sizeof(unsigned long long), c->stream));
  }
  DecompArgs A;
  A.teams = dteams.as<Team>();
  A.nteams = nteams;
  A.team_words = words.as<DevWords>();
  A.off = g.off.as<uint64_t>();
  A.adj = g.adj.as<uint32_t>();
  A.deg = deg.as<uint32_t>();
  A.rem = rem.as<uint32_t>();
  A.core = dcore;
  A.list[0] = alive.as<uint32_t>();
  A.list[1] = list2.as<uint32_t>();
  A.cand[0] = cand0.as<uint32_t>();
  A.cand[1] = cand1.as<uint32_t>();
  A.front[0] = front[0].as<uint32_t>();
  A.front[1] = front[1].as<uint32_t>();
  A.big = big.as<uint32_t>();
  A.cnt = cn.as<unsigned long long>();
  A.n_list = n_alive;
  A.cap = n;
  A.big_row = big_row(c);
  A.window = (uint32_t)std::min<int64_t>(std::max<int64_t>(1, c->opt.kcore_window), 1 << 20);
  A.words = dev_words(c);
  A.timeout_ns = (unsigned long long)c->opt.timeout_ms * 1000000ULL;
  void* p[] = {&A};
  uint64_t h[5] = {};
  {
    CoopLock coop(c);
    const void* kernel = teams.empty() ? (const void*)k_core_levels<false> : (const void*)k_core_levels<true>;
    KT_CUDA(cudaLaunchCooperativeKernel(kernel, dim3(grid), dim3(kCoreThreads), p, 0,
                                        c->stream));
    KT_LAUNCHED(c);
    if (!teams.empty()) {
      merge_team_errors(c, words.get(), nteams);
    }
    if (teams.empty()) {
      copy_d2h(c, h, cn.as<unsigned long long>() + 14, sizeof(h));
    } else {  // the most of each
      std::vector<unsigned long long> all(nteams * kTeamCounters);
      copy_d2h(c, all.data(), cn.get(), all.size() * sizeof(unsigned long long));
      for (unsigned t = 0; t < nteams; ++t)
        for (int q = 0; q < 5; ++q) h[q] = std::max<uint64_t>(h[q], all[t * kTeamCounters + 14 + q]);
    }
  }
  rounds += h[0];
  probes += h[1];
  check_words(c, "core decomposition");
  KT_LOG(c,
         "kt: core decomposition of %llu vertices by %u teams: %llu levels, %llu rounds, %llu passes (%llu full), "
         "max core %llu\n",
         (unsigned long long)n_alive, nteams, (unsigned long long)h[1], (unsigned long long)h[0],
         (unsigned long long)h[2],
         (unsigned long long)h[3], (unsigned long long)(h[4] ? h[4] - 1 : 0));
  n_alive = 0;  // the state is consumed
}

}  // namespace kt
