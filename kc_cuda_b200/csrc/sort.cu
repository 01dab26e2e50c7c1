// Stable LSD radix sort of 64-bit keys (optionally carrying a 32-bit value) by
// chosen bit fields, digits of at most 8 bits.
//
// One pass = tile histograms -> digit-major exclusive scan -> stable scatter:
// a tile of kSortTile keys ranks them (each warp owns consecutive keys and
// finds the lanes with a key's digit by a ballot per bit, against warp-private
// running digit counters), places the tile in shared memory sorted by digit and writes every
// digit's run with consecutive threads on consecutive addresses.  (Counting
// all passes at once and finding each tile's places by look-back over the tiles
// before it, one word per digit and tile, reads the keys once less but was
// slower, 113 against 100 us a pass of 16M keys: the words are an eighth of the
// keys' bytes, read several times over.)  At most one tile of keys is sorted in
// shared memory by one block in one launch.
//
// The scatter is bound by the shared-memory pipe (87 % busy, DRAM 24 %, with the
// lanes matched by __match_any_sync, which is the slower the more digits a warp
// has): 1.05-1.14 ms a pass of 214M random keys by ballots, 1.26-1.39 by match;
// taking places by atomics of the first lane instead of a load and a store:
// 1.10-1.20.
#include <algorithm>

#include "kt_device.cuh"
#include "kt_internal.h"

namespace kt {
namespace {

// (16 keys per lane in 256 threads, three blocks per SM: 13.5 ms over the 60
// scatters of a batch of 64 mix graphs; 4 blocks spill and take 14.8, 512
// threads 15.0 to 15.7, 24 keys per lane 16.8.)
constexpr unsigned kSortThreads = 256;
constexpr unsigned kSortWarps = kSortThreads / 32;
constexpr unsigned kSortIpt = 16;    // keys per lane
constexpr unsigned kSortBlocks = 3;  // resident blocks per SM
constexpr unsigned kWarpKeys = 32 * kSortIpt;
constexpr unsigned kSortTile = kSortWarps * kWarpKeys;
constexpr int kMaxPasses = 10;

struct Digits {
  int passes;
  int shift[kMaxPasses];
  uint32_t mask[kMaxPasses];
};

__global__ void __launch_bounds__(kSortThreads) k_tile_hist(const uint64_t* __restrict__ keys, uint64_t n, int shift,
                                                            uint32_t mask, uint32_t ntiles,
                                                            uint32_t* __restrict__ tile_hist) {
  __shared__ uint32_t h[256];
  if (threadIdx.x < 256) h[threadIdx.x] = 0;
  __syncthreads();
  const uint64_t base = (uint64_t)blockIdx.x * kSortTile;
#pragma unroll 8
  for (unsigned i = 0; i < kSortIpt; ++i) {
    const uint64_t j = base + i * kSortThreads + threadIdx.x;
    if (j < n) atomicAdd(&h[(uint32_t)(keys[j] >> shift) & mask], 1u);
  }
  __syncthreads();
  if (threadIdx.x <= mask) tile_hist[(uint64_t)threadIdx.x * ntiles + blockIdx.x] = h[threadIdx.x];
}

struct SortShared {
  uint32_t wrun[kSortWarps][256];  // running counts per warp and digit, then the warps' first places in the tile
  uint32_t dstart[256];            // the digits' first places in the tile
  uint32_t tmp[33];
};

// Ranks the tile's keys k[] (entry j of lane l of warp w is key w * kWarpKeys +
// j * 32 + l, valid below tn) by a digit: on return rank[] is each key's place in
// its warp's run of the digit, S.wrun the warps' first places of it in the tile,
// S.dstart the digits' first places.
__device__ __forceinline__ void rank_tile(SortShared& S, const uint64_t (&k)[kSortIpt], uint32_t tn, int shift,
                                              uint32_t mask, uint32_t (&rank)[kSortIpt]) {
  const unsigned w = warp_id(), l = lane_id();
  for (unsigned q = threadIdx.x; q < kSortWarps * 256; q += kSortThreads) (&S.wrun[0][0])[q] = 0;
  __syncthreads();
  const unsigned lt = lanemask_lt();
#pragma unroll
  for (unsigned j = 0; j < kSortIpt; ++j) {
    const bool valid = w * kWarpKeys + j * 32 + l < tn;
    const uint32_t d = (uint32_t)(k[j] >> shift) & mask;
    unsigned peers = __ballot_sync(kFull, valid);
#pragma unroll
    for (unsigned b = 0; b < 8; ++b) {
      if (!((mask >> b) & 1)) break;  // (a mask of low bits)
      const unsigned have = __ballot_sync(kFull, (d >> b) & 1);
      peers &= (d >> b) & 1 ? have : ~have;
    }
    const uint32_t base = valid ? S.wrun[w][d] : 0u;
    __syncwarp();
    if (valid && l == (unsigned)(__ffs(peers) - 1)) S.wrun[w][d] = base + __popc(peers);
    __syncwarp();
    rank[j] = base + __popc(peers & lt);
  }
  __syncthreads();
  // One digit a thread: its first place, then the warps' places after it.
  const unsigned d = threadIdx.x;
  uint32_t s = 0;
#pragma unroll
  for (unsigned q = 0; q < kSortWarps; ++q) s += S.wrun[q][d];
  uint32_t total;
  s = block_excl_scan<uint32_t>(s, S.tmp, &total);
  S.dstart[d] = s;
#pragma unroll
  for (unsigned q = 0; q < kSortWarps; ++q) {
    const uint32_t t = S.wrun[q][d];
    S.wrun[q][d] = s;
    s += t;
  }
  __syncthreads();
}
static_assert(kSortThreads == 256, "a thread per digit");

template <bool kVals>
__device__ __forceinline__ void place_tile(const SortShared& S, const uint64_t (&k)[kSortIpt],
                                           const uint32_t (&v)[kSortIpt], const uint32_t (&rank)[kSortIpt],
                                           uint32_t tn, int shift, uint32_t mask, uint64_t* skeys, uint32_t* svals) {
  const unsigned w = warp_id(), l = lane_id();
#pragma unroll
  for (unsigned j = 0; j < kSortIpt; ++j) {
    if (w * kWarpKeys + j * 32 + l < tn) {
      const uint32_t d = (uint32_t)(k[j] >> shift) & mask;
      const uint32_t p = S.wrun[w][d] + rank[j];
      skeys[p] = k[j];
      if (kVals) svals[p] = v[j];
    }
  }
  __syncthreads();
}

// Scatter of one tile by the digit (key >> shift) & mask; tile_off: the first
// place of each (digit, tile).  kCheck: nothing is written; each key is compared
// with the one that `want` has in its place, and *bad set where they differ.
template <bool kVals, bool kCheck>
__global__ void __launch_bounds__(kSortThreads, kSortBlocks) k_scatter(const uint64_t* __restrict__ keys,
                                                          const uint32_t* __restrict__ vals, uint64_t n, int shift,
                                                          uint32_t mask, uint32_t ntiles,
                                                          const uint32_t* __restrict__ tile_off,
                                                          uint64_t* __restrict__ keys_out,
                                                          uint32_t* __restrict__ vals_out,
                                                          const uint64_t* __restrict__ want,
                                                          uint32_t* __restrict__ bad) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  uint64_t* skeys = reinterpret_cast<uint64_t*>(smem_raw);                  // kSortTile
  uint32_t* svals = reinterpret_cast<uint32_t*>(smem_raw + kSortTile * 8);  // kSortTile (kVals)
  __shared__ SortShared S;
  __shared__ uint32_t toff[256];
  const unsigned w = warp_id(), l = lane_id();
  const uint64_t tbase = (uint64_t)blockIdx.x * kSortTile;
  const uint32_t tn = (uint32_t)(n - tbase < kSortTile ? n - tbase : kSortTile);
  uint64_t k[kSortIpt];
  uint32_t v[kSortIpt];
  uint32_t rank[kSortIpt];
#pragma unroll
  for (unsigned j = 0; j < kSortIpt; ++j) {
    const uint32_t at = w * kWarpKeys + j * 32 + l;
    k[j] = at < tn ? keys[tbase + at] : 0;
    if (kVals) v[j] = at < tn ? vals[tbase + at] : 0;
  }
  if (threadIdx.x <= mask) toff[threadIdx.x] = tile_off[(uint64_t)threadIdx.x * ntiles + blockIdx.x];
  rank_tile(S, k, tn, shift, mask, rank);
  place_tile<kVals>(S, k, v, rank, tn, shift, mask, skeys, svals);
  for (uint32_t i = threadIdx.x; i < tn; i += kSortThreads) {
    const uint64_t key = skeys[i];
    const uint32_t q = (uint32_t)(key >> shift) & mask;
    const uint32_t pos = toff[q] + (i - S.dstart[q]);
    if (kCheck) {
      if (want[pos] != key) *bad = 1u;
    } else {
      keys_out[pos] = key;
      if (kVals) vals_out[pos] = svals[i];
    }
  }
}

// keys[0..n) against want[0..n).
__global__ void k_equal_u64(const uint64_t* __restrict__ keys, const uint64_t* __restrict__ want, uint64_t n,
                            uint32_t* __restrict__ bad) {
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x)
    if (keys[i] != want[i]) *bad = 1u;
}

// All passes of at most one tile, in place.
template <bool kVals>
__global__ void __launch_bounds__(kSortThreads) k_sort_tile(uint64_t* __restrict__ keys, uint32_t* __restrict__ vals,
                                                            uint32_t n, Digits D) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  uint64_t* skeys = reinterpret_cast<uint64_t*>(smem_raw);
  uint32_t* svals = reinterpret_cast<uint32_t*>(smem_raw + kSortTile * 8);
  __shared__ SortShared S;
  const unsigned w = warp_id(), l = lane_id();
  uint64_t k[kSortIpt];
  uint32_t v[kSortIpt];
  uint32_t rank[kSortIpt];
#pragma unroll
  for (unsigned j = 0; j < kSortIpt; ++j) {
    const uint32_t at = w * kWarpKeys + j * 32 + l;
    k[j] = at < n ? keys[at] : 0;
    if (kVals) v[j] = at < n ? vals[at] : 0;
  }
  for (int p = 0; p < D.passes; ++p) {
    rank_tile(S, k, n, D.shift[p], D.mask[p], rank);
    place_tile<kVals>(S, k, v, rank, n, D.shift[p], D.mask[p], skeys, svals);
#pragma unroll
    for (unsigned j = 0; j < kSortIpt; ++j) {
      const uint32_t at = w * kWarpKeys + j * 32 + l;
      if (at < n) {
        k[j] = skeys[at];
        if (kVals) v[j] = svals[at];
      }
    }
    __syncthreads();
  }
#pragma unroll
  for (unsigned j = 0; j < kSortIpt; ++j) {
    const uint32_t at = w * kWarpKeys + j * 32 + l;
    if (at < n) {
      keys[at] = k[j];
      if (kVals) vals[at] = v[j];
    }
  }
}

}  // namespace

static void sort_passes(Ctx* c, uint64_t* keys, uint32_t* vals, uint64_t n, std::initializer_list<BitField> fields,
                        const uint64_t* want, uint32_t* bad) {
  auto compare = [&] {
    if (!want || !n) return;
    k_equal_u64<<<grid_for(n, 256, c->num_sms * 16), 256, 0, c->stream>>>(keys, want, n, bad);
    KT_LAUNCHED(c);
  };
  Digits D{};
  for (const BitField& f : fields) {
    // Digits of equal width, at most 8 bits each.
    const int bits = std::min(f.hi, 64) - f.lo, parts = (bits + 7) / 8;
    for (int i = 0; i < parts; ++i) {
      const int lo = f.lo + bits * i / parts, hi = f.lo + bits * (i + 1) / parts;
      if (D.passes == kMaxPasses) throw Error(KT_ERR_CUDA, "radix sort: too many passes");
      D.shift[D.passes] = lo;
      D.mask[D.passes++] = (1u << (hi - lo)) - 1;
    }
  }
  if (n < 2 || D.passes == 0) {
    compare();
    return;
  }
  if (n >= 0xffffffffULL) throw Error(KT_ERR_LIMIT, "radix sort: more than 2^32-1 keys");
  const size_t smem = kSortTile * (vals ? 12 : 8);
  if (n <= kSortTile) {
    if (vals) {
      allow_max_dynamic_smem((const void*)k_sort_tile<true>);
      k_sort_tile<true><<<1, kSortThreads, smem, c->stream>>>(keys, vals, (uint32_t)n, D);
    } else {
      allow_max_dynamic_smem((const void*)k_sort_tile<false>);
      k_sort_tile<false><<<1, kSortThreads, smem, c->stream>>>(keys, nullptr, (uint32_t)n, D);
    }
    KT_LAUNCHED(c);
    compare();
    return;
  }
  const uint32_t ntiles = (uint32_t)((n + kSortTile - 1) / kSortTile);
  allow_max_dynamic_smem((const void*)k_scatter<true, false>);
  allow_max_dynamic_smem((const void*)k_scatter<false, false>);
  allow_max_dynamic_smem((const void*)k_scatter<false, true>);
  DBuf keys_alt(c, n * sizeof(uint64_t));
  DBuf vals_alt;
  if (vals) vals_alt.alloc(c, n * sizeof(uint32_t));
  DBuf th(c, (uint64_t)ntiles * 256 * sizeof(uint32_t));
  uint64_t* ksrc = keys;
  uint64_t* kdst = keys_alt.as<uint64_t>();
  uint32_t* vsrc = vals;
  uint32_t* vdst = vals ? vals_alt.as<uint32_t>() : nullptr;
  for (int p = 0; p < D.passes; ++p) {
    k_tile_hist<<<ntiles, kSortThreads, 0, c->stream>>>(ksrc, n, D.shift[p], D.mask[p], ntiles, th.as<uint32_t>());
    KT_LAUNCHED(c);
    scan_u32(c, th.as<uint32_t>(), th.as<uint32_t>(), (uint64_t)ntiles * (D.mask[p] + 1));
    if (want && p + 1 == D.passes) {
      k_scatter<false, true><<<ntiles, kSortThreads, smem, c->stream>>>(ksrc, nullptr, n, D.shift[p], D.mask[p], ntiles,
                                                                        th.as<uint32_t>(), nullptr, nullptr, want, bad);
      KT_LAUNCHED(c);
      return;
    }
    if (vals)
      k_scatter<true, false><<<ntiles, kSortThreads, smem, c->stream>>>(ksrc, vsrc, n, D.shift[p], D.mask[p], ntiles,
                                                                        th.as<uint32_t>(), kdst, vdst, nullptr, nullptr);
    else
      k_scatter<false, false><<<ntiles, kSortThreads, smem, c->stream>>>(ksrc, nullptr, n, D.shift[p], D.mask[p],
                                                                         ntiles, th.as<uint32_t>(), kdst, nullptr,
                                                                         nullptr, nullptr);
    KT_LAUNCHED(c);
    std::swap(ksrc, kdst);
    std::swap(vsrc, vdst);
  }
  if (ksrc != keys) {
    KT_CUDA(cudaMemcpyAsync(keys, ksrc, n * sizeof(uint64_t), cudaMemcpyDeviceToDevice, c->stream));
    if (vals) KT_CUDA(cudaMemcpyAsync(vals, vsrc, n * sizeof(uint32_t), cudaMemcpyDeviceToDevice, c->stream));
  }
}

void radix_sort_u64(Ctx* c, uint64_t* keys, uint32_t* vals, uint64_t n, std::initializer_list<BitField> fields) {
  sort_passes(c, keys, vals, n, fields, nullptr, nullptr);
}

void radix_sort_compare(Ctx* c, uint64_t* keys, uint64_t n, std::initializer_list<BitField> fields,
                        const uint64_t* want, uint32_t* bad) {
  sort_passes(c, keys, nullptr, n, fields, want, bad);
}

}  // namespace kt
