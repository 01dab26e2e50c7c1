// Order-preserving stream compaction of an index range by a predicate, in one
// pass: a tile of 2048 indices evaluates the predicate once per index (rows of
// 256 indices, so its loads are coalesced), numbers the kept ones by warp
// ballots, finds its prefix by look-back and writes their values.  No n-sized
// temporaries.
#pragma once
#include "kt_device.cuh"
#include "kt_internal.h"
#include "lookback.cuh"
#include "stages.h"

namespace kt {

constexpr unsigned kCompactThreads = 256;
constexpr unsigned kCompactItems = 8;
constexpr unsigned kCompactTile = kCompactThreads * kCompactItems;

Lookback begin_lookback(Ctx* c, uint64_t tiles);
void end_lookback(Ctx* c, uint64_t tiles);

template <class F, typename T>
__global__ void __launch_bounds__(kCompactThreads, 8) k_compact(uint64_t n, F f, T* __restrict__ out, Lookback L,
                                                             unsigned long long* __restrict__ count) {
  constexpr unsigned kWarps = kCompactThreads / 32;
  __shared__ uint32_t first[kCompactItems * kWarps];  // kept before each (row, warp) of the tile
  __shared__ unsigned long long sh[2];
  const uint64_t tile = gridDim.x > 1 ? take_tile(L, &sh[0]) : 0;
  if (tile >= gridDim.x) return;
  const uint64_t base = tile * kCompactTile;
  const unsigned w = warp_id(), lane = lane_id();
  unsigned kept[kCompactItems];
  bool keep[kCompactItems];
#pragma unroll
  for (unsigned i = 0; i < kCompactItems; ++i) {
    const uint64_t j = base + i * kCompactThreads + threadIdx.x;
    keep[i] = j < n && f.keep(j);
  }
#pragma unroll
  for (unsigned i = 0; i < kCompactItems; ++i) {
    kept[i] = __ballot_sync(kFull, keep[i]);
    if (lane == 0) first[i * kWarps + w] = __popc(kept[i]);
  }
  __syncthreads();
  if (w == 0) {
    static_assert(kCompactItems * kWarps == 64, "two counts per lane");
    const uint32_t a = first[2 * lane], b = first[2 * lane + 1];
    const uint32_t incl = warp_incl_scan(a + b);
    const uint32_t own = __shfl_sync(kFull, incl, 31);
    __syncwarp();
    first[2 * lane] = incl - a - b;
    first[2 * lane + 1] = incl - b;
    unsigned long long p = 0;
    if (gridDim.x > 1)
      p = tile_prefix(L, tile, own, false, [&](uint64_t t) {
        unsigned long long s = 0;
#pragma unroll 1
        for (unsigned i = lane; i < kCompactTile; i += 32)
          s += t * kCompactTile + i < n && f.keep(t * kCompactTile + i);
        return warp_sum(s);
      });
    if (lane == 0) {
      sh[1] = p;
      if (tile == gridDim.x - 1) *count = p + own;
    }
  }
  __syncthreads();
  const uint64_t at = sh[1];
#pragma unroll
  for (unsigned i = 0; i < kCompactItems; ++i)
    if (keep[i])
      out[at + first[i * kWarps + w] + __popc(kept[i] & lanemask_lt())] =
          f.value(base + i * kCompactThreads + threadIdx.x);
}

// Returns the number of kept items; out receives f.value(i) for each kept i
// in increasing i.
template <class F, typename T>
uint64_t compact(Ctx* c, uint64_t n, const F& f, T* out) {
  if (n == 0) return 0;
  const uint64_t tiles = (n + kCompactTile - 1) / kCompactTile;
  if (tiles > 0x7fffffffULL) throw Error(KT_ERR_LIMIT, "compaction: too many tiles");
  const Lookback L = begin_lookback(c, tiles);
  unsigned long long* count = c->lb_ticket.as<unsigned long long>() + 1;
  k_compact<F, T><<<(unsigned)tiles, kCompactThreads, 0, c->stream>>>(n, f, out, L, count);
  KT_LAUNCHED(c);
  if (tiles > 1) end_lookback(c, tiles);
  return read_word<unsigned long long>(c, count);
}

}  // namespace kt
