// Device-wide scans and the sorted-unique compaction.
//
// Scans and compactions (compact.cuh) take one pass over the data in one
// launch: tiles of 2048 items (256 threads x 8) find their prefix by decoupled
// look-back.  (Tile sums, a recursive scan of those and a second pass over the
// data took three to seven launches, most of the small kernels of a solve:
// R-MAT scale 10, 1.65 -> 1.37 ms with one.)
#include "compact.cuh"
#include "kt_device.cuh"
#include "kt_internal.h"
#include "lookback.cuh"

namespace kt {

// The context's look-back words for one launch of `tiles` tiles.
Lookback begin_lookback(Ctx* c, uint64_t tiles) {
  if (!c->lb_ticket.get()) {
    c->lb_ticket.alloc(c, 2 * sizeof(unsigned long long));  // the ticket, and a launch's total
    zero(c, c->lb_ticket.get(), c->lb_ticket.bytes());
    c->lb_tickets = 0;
  }
  if (c->lb_status.bytes() < tiles * sizeof(unsigned long long) || ++c->lb_epoch >= kEpochs) {
    c->lb_status.ensure(c, std::max<uint64_t>(tiles, 1 << 9) * sizeof(unsigned long long));
    zero(c, c->lb_status.get(), c->lb_status.bytes());
    c->lb_epoch = 1;
  }
  return Lookback{c->lb_status.as<unsigned long long>(), c->lb_ticket.as<unsigned long long>(), c->lb_tickets,
                  c->lb_epoch,
                  std::min((unsigned long long)c->opt.timeout_ms * 1000000ULL, kTileWaitNs)};
}
void end_lookback(Ctx* c, uint64_t tiles) { c->lb_tickets += tiles; }

namespace {

constexpr unsigned kScanThreads = 256;
constexpr unsigned kScanItems = 8;
constexpr unsigned kScanTile = kScanThreads * kScanItems;

// Exclusive scan.  In-place safe (out is in, or they are apart): a tile is read
// before any of it is written.
template <typename Tin, typename Tout>
__global__ void __launch_bounds__(kScanThreads, 6) k_scan(const Tin* in, Tout* out, uint64_t n, Lookback L) {
  __shared__ Tout stage[kScanTile];
  __shared__ Tout tmp[33];
  __shared__ unsigned long long sh[2];
  const uint64_t tile = gridDim.x > 1 ? take_tile(L, &sh[0]) : 0;
  if (tile >= gridDim.x) return;
  const uint64_t base = tile * kScanTile;
#pragma unroll
  for (unsigned i = 0; i < kScanItems; ++i) {
    const uint64_t j = base + i * kScanThreads + threadIdx.x;
    stage[i * kScanThreads + threadIdx.x] = j < n ? (Tout)in[j] : Tout(0);
  }
  __syncthreads();
  Tout v[kScanItems];
  Tout run = 0;
#pragma unroll
  for (unsigned i = 0; i < kScanItems; ++i) {
    v[i] = run;
    run += stage[threadIdx.x * kScanItems + i];
  }
  Tout total;
  const Tout excl = block_excl_scan<Tout>(run, tmp, &total);
  if (gridDim.x > 1) {
    if (warp_id() == 0) {
      const bool in_place = (const void*)in == (const void*)out;
      const unsigned long long p = tile_prefix(L, tile, (unsigned long long)total, in_place, [&](uint64_t t) {
        const volatile Tin* from = in + t * kScanTile;
        Tout s = 0;
#pragma unroll 1
        for (unsigned i = lane_id(); i < kScanTile; i += 32) s += (Tout)(t * kScanTile + i < n ? from[i] : Tin(0));
        return (unsigned long long)warp_sum(s);
      });
      if (lane_id() == 0) sh[1] = p;
    }
  } else if (threadIdx.x == 0) {
    sh[1] = 0;
  }
  __syncthreads();
  const Tout off = (Tout)sh[1] + excl;
#pragma unroll
  for (unsigned i = 0; i < kScanItems; ++i) stage[threadIdx.x * kScanItems + i] = v[i] + off;
  __syncthreads();
#pragma unroll
  for (unsigned i = 0; i < kScanItems; ++i) {
    const uint64_t j = base + i * kScanThreads + threadIdx.x;
    if (j < n) out[j] = stage[i * kScanThreads + threadIdx.x];
  }
}

template <typename Tin, typename Tout>
void scan_impl(Ctx* c, const Tin* in, Tout* out, uint64_t n) {
  if (n == 0) return;
  const uint64_t tiles = (n + kScanTile - 1) / kScanTile;
  if (tiles > 0x7fffffffULL) throw Error(KT_ERR_LIMIT, "scan: too many tiles");
  const Lookback L = tiles > 1 ? begin_lookback(c, tiles) : Lookback{};
  k_scan<Tin, Tout><<<(unsigned)tiles, kScanThreads, 0, c->stream>>>(in, out, n, L);
  KT_LAUNCHED(c);
  if (tiles > 1) end_lookback(c, tiles);
}

// Distinct keys of a sorted list, ~0 dropped.
struct DistinctKey {
  const uint64_t* in;
  __device__ bool keep(uint64_t j) const {
    const uint64_t k = in[j];
    return k != ~0ULL && (j == 0 || in[j - 1] != k);
  }
  __device__ uint64_t value(uint64_t j) const { return in[j]; }
};

}  // namespace

void scan_u32(Ctx* c, const uint32_t* in, uint32_t* out, uint64_t n) { scan_impl<uint32_t, uint32_t>(c, in, out, n); }
void scan_u32_to_u64(Ctx* c, const uint32_t* in, uint64_t* out, uint64_t n) { scan_impl<uint32_t, uint64_t>(c, in, out, n); }

uint64_t unique_sorted_u64(Ctx* c, const uint64_t* in, uint64_t* out, uint64_t n) {
  return compact(c, n, DistinctKey{in}, out);
}

}  // namespace kt
