// Decoupled look-back: the running sum over the tiles of one launch, in one
// pass over the data (tiles publish their own sum, then look back over their
// predecessors' until one has published its running sum).
//
// A status word holds flag (2 bits), epoch (14 bits) and value (48 bits), so one
// 64-bit load tells whether it is this pass's and what it says; words of
// earlier passes need no clearing.  Tiles are numbered by a ticket taken when
// the block starts, so a tile only waits for blocks that are already running.
// Waits are bounded: past the bound kDevErrWait is flagged and the tile writes
// nothing.
#pragma once
#include "kt_device.cuh"

namespace kt {

constexpr unsigned long long kTileSum = 1ULL << 62, kTilePrefix = 2ULL << 62;
constexpr unsigned long long kTileValue = (1ULL << 48) - 1;
constexpr uint32_t kEpochs = 1u << 14;  // epochs 1 .. kEpochs - 1 are used
constexpr uint32_t kLookbackPolls = 1u << 22;

struct Lookback {
  unsigned long long* status;  // one word per tile (times the digits, in a sort)
  unsigned long long* ticket;  // counts the tiles of every launch so far
  unsigned long long base;     // its value before this launch
  uint32_t epoch;
  uint32_t* err;
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
  for (uint32_t i = 0; i < kLookbackPolls; ++i) {
    const unsigned long long v = ld_relaxed_u64(p);
    if (((v >> 48) & (kEpochs - 1)) == L.epoch) return v;
    if (i > 64) __nanosleep(64);
  }
  atomicOr(L.err, kDevErrWait);
  return 0;
}

// This block's tile.  Every thread of the block calls it, and leaves when the
// tile is not one of the launch's.
__device__ __forceinline__ uint64_t take_tile(const Lookback& L, unsigned long long* sh) {
  if (threadIdx.x == 0) *sh = atomicAdd(L.ticket, 1ULL) - L.base;
  __syncthreads();
  return *sh;
}

// Sum of the tiles before `tile`, whose own sum is `own`; *ok false when a wait
// gave up.  Called by one whole warp.
__device__ __forceinline__ unsigned long long tile_prefix(const Lookback& L, uint64_t tile, unsigned long long own,
                                                          bool* ok) {
  const unsigned lane = lane_id();
  if (tile == 0) {
    if (lane == 0) st_relaxed_u64(&L.status[0], tile_word(kTilePrefix, L.epoch, own));
    *ok = true;
    return 0;
  }
  if (lane == 0) st_relaxed_u64(&L.status[tile], tile_word(kTileSum, L.epoch, own));
  unsigned long long sum = 0;
  for (int64_t last = (int64_t)tile - 1;; last -= 32) {
    const int64_t p = last - lane;
    const unsigned long long w = p >= 0 ? wait_tile_word(L, &L.status[p]) : kTilePrefix;
    if (__any_sync(kFull, w == 0)) {
      *ok = false;
      return 0;
    }
    const unsigned done = __ballot_sync(kFull, (w & kTilePrefix) != 0);
    const unsigned upto = done ? (unsigned)__ffs(done) - 1 : 31u;
    sum += warp_sum(lane <= upto ? (w & kTileValue) : 0ULL);
    if (done) break;
  }
  if (lane == 0) st_relaxed_u64(&L.status[tile], tile_word(kTilePrefix, L.epoch, sum + own));
  *ok = true;
  return sum;
}

}  // namespace kt
