// Decoupled look-back: the running sum over the tiles of one launch, in one
// pass over the data (tiles publish their own sum, then look back over their
// predecessors' until one has published its running sum).
//
// A status word holds flag (2 bits), epoch (14 bits) and value (48 bits), so one
// 64-bit load tells whether it is this pass's and what it says; words of
// earlier passes need no clearing.  Tiles are numbered by a ticket taken when
// the block starts, so a tile only waits for blocks that are already running.
// Waits are bounded, and what a wait was for can be had without it: past the
// bound the tile adds up its predecessor's items itself.  So a pass always ends
// with the right sums, and nothing after it has to ask whether it did.
#pragma once
#include "kt_device.cuh"

namespace kt {

constexpr unsigned long long kTileSum = 1ULL << 62, kTilePrefix = 2ULL << 62;
constexpr unsigned long long kTileValue = (1ULL << 48) - 1;
constexpr uint32_t kEpochs = 1u << 14;  // epochs 1 .. kEpochs - 1 are used
constexpr unsigned long long kTileWaitNs = 10000000ULL;  // (a tile normally waits microseconds)

struct Lookback {
  unsigned long long* status;  // one word per tile (times the digits, in a sort)
  unsigned long long* ticket;  // counts the tiles of every launch so far
  unsigned long long base;     // its value before this launch
  uint32_t epoch;
  unsigned long long wait_ns;  // bound on a wait for one predecessor
};

__device__ __forceinline__ unsigned long long tile_word(unsigned long long flag, uint32_t epoch,
                                                        unsigned long long v) {
  return flag | ((unsigned long long)epoch << 48) | v;
}
__device__ __forceinline__ void st_relaxed_u64(unsigned long long* p, unsigned long long v) {
  asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}

// The word at p once it belongs to this epoch; 0 when the wait gave up.
__device__ __forceinline__ unsigned long long wait_tile_word(const Lookback& L, const unsigned long long* p) {
  unsigned long long t0 = 0;
  for (uint32_t i = 0;; ++i) {
    const unsigned long long v = ld_relaxed_u64(p);
    if (((v >> 48) & (kEpochs - 1)) == L.epoch) return v;
    if (L.wait_ns == 0) return 0;
    if (i >= 64) {
      if ((i & 63) == 0) {
        const unsigned long long now = globaltimer_ns();
        if (!t0) t0 = now;
        if (now - t0 >= L.wait_ns) return 0;
      }
      __nanosleep(64);
    }
  }
}

// This block's tile.  Every thread of the block calls it, and leaves when the
// tile is not one of the launch's.
__device__ __forceinline__ uint64_t take_tile(const Lookback& L, unsigned long long* sh) {
  if (threadIdx.x == 0) *sh = atomicAdd(L.ticket, 1ULL) - L.base;
  __syncthreads();
  return *sh;
}

// Sum of the tiles before `tile`, whose own sum is `own`.  Called by one whole
// warp; sum_of(p) is the sum of tile p's items, found by the whole warp from the
// input.  Where the output may overwrite the input (`in_place`), a tile does so
// after its word is out, so items read before the word was seen missing are the
// input's.
template <class Sum>
__device__ __forceinline__ unsigned long long tile_prefix(const Lookback& L, uint64_t tile, unsigned long long own,
                                                          bool in_place, Sum sum_of) {
  const unsigned lane = lane_id();
  if (lane == 0) {
    st_relaxed_u64(&L.status[tile], tile_word(tile ? kTileSum : kTilePrefix, L.epoch, own));
    if (in_place) __threadfence();  // (before the block's writes, which follow a block barrier)
  }
  if (tile == 0) return 0;
  unsigned long long sum = 0;
  for (int64_t last = (int64_t)tile - 1;; last -= 32) {
    const int64_t p = last - lane;
    unsigned long long w = p >= 0 ? wait_tile_word(L, &L.status[p]) : kTilePrefix;
    __syncwarp();
    unsigned done = __ballot_sync(kFull, (w & kTilePrefix) != 0);
    unsigned late = __ballot_sync(kFull, w == 0);
    if (done) late &= (done & -done) - 1;  // those that count
    while (late) {
      const unsigned l = __ffs(late) - 1;
      late &= late - 1;
      const unsigned long long s = sum_of((uint64_t)(last - l)) & kTileValue;
      __threadfence();
      __syncwarp();
      if (lane == l) {
        w = ld_relaxed_u64(&L.status[p]);
        if (((w >> 48) & (kEpochs - 1)) != L.epoch) w = tile_word(kTileSum, L.epoch, s);
      }
    }
    done = __ballot_sync(kFull, (w & kTilePrefix) != 0);
    const unsigned upto = done ? (unsigned)__ffs(done) - 1 : 31u;
    sum += warp_sum(lane <= upto ? (w & kTileValue) : 0ULL);
    if (done) break;
  }
  if (lane == 0) st_relaxed_u64(&L.status[tile], tile_word(kTilePrefix, L.epoch, sum + own));
  return sum;
}

}  // namespace kt
