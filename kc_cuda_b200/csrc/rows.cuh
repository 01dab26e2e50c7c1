// Adjacency rows read by a whole grid: windows of long rows dealt to every
// warp, and the filtered, renumbered copy of a list of rows (the compaction of
// a core, the entries of a working subgraph).
#pragma once
#include "compact.cuh"
#include "kt_device.cuh"
#include "kt_internal.h"

namespace kt {

constexpr unsigned kBigBatch = 1024;  // long rows per batch of dealt windows

// Deals the kWin-entry windows of the rows row(0), ..., row(nbig - 1) of
// `off` to every warp of the grid (or crew), so one long row is spread over the whole
// GPU instead of one block: each block lists the rows' first window numbers
// (the same block scan in every block, kBigBatch rows at a time) and warp w
// takes windows w, w + warps, ...; `drop(i, b, e)` handles entries [b, e) (at
// most kWin) of row(i).  Every thread of the block must call it (it
// synchronises the block); blocks have 256, 512 or 1024 threads.
template <unsigned kWin, class Row, class Drop>
__device__ __forceinline__ void deal_windows(uint64_t nbig, Row row, const uint64_t* __restrict__ off, uint64_t* woff,
                                             uint64_t* tmp, Drop drop, Crew crew = Crew()) {
  const uint64_t gwarps = (uint64_t)crew.blocks * (blockDim.x >> 5);
  const uint64_t gwarp = (uint64_t)crew.rank * (blockDim.x >> 5) + warp_id();
  constexpr unsigned kMost = kBigBatch / 256;
  const unsigned per = kBigBatch / blockDim.x;  // rows per thread
  for (uint64_t base = 0; base < nbig; base += kBigBatch) {
    const uint64_t left = nbig - base;
    const uint32_t cnt = left < kBigBatch ? (uint32_t)left : kBigBatch;
    uint64_t w[kMost];
    uint64_t sum = 0;
#pragma unroll
    for (unsigned j = 0; j < kMost; ++j) {
      const uint32_t r = threadIdx.x * per + j;
      w[j] = 0;
      if (j < per && r < cnt) {
        const uint32_t v = row(base + r);
        w[j] = (off[v + 1] - off[v] + kWin - 1) / kWin;
      }
      sum += w[j];
    }
    uint64_t total;
    uint64_t pre = block_excl_scan<uint64_t>(sum, tmp, &total);
#pragma unroll
    for (unsigned j = 0; j < kMost; ++j) {
      const uint32_t r = threadIdx.x * per + j;
      if (j < per && r < cnt) woff[r] = pre;
      pre += w[j];
    }
    if (threadIdx.x == 0) woff[cnt] = total;
    __syncthreads();
    for (uint64_t x = gwarp; x < total; x += gwarps) {
      uint32_t lo = 0, hi = cnt;  // last row with woff <= x
      while (hi - lo > 1) {
        const uint32_t mid = (lo + hi) >> 1;
        if (woff[mid] <= x)
          lo = mid;
        else
          hi = mid;
      }
      const uint32_t v = row(base + lo);
      const uint64_t b = off[v] + (x - woff[lo]) * kWin, e = min(off[v + 1], b + kWin);
      drop(base + lo, b, e);
    }
    __syncthreads();
  }
}

// Rows of more than kLongRow entries are copied by the whole grid.  A warp
// reads 128 entries at a step, so the line is four steps of one warp; beyond
// it a hub row is a serial chain: with a warp per row of any length the working
// subgraphs of an R-MAT scale 22 graph (rows of up to a few hundred thousand
// entries) took 6.5 ms of a 48.6 ms solve.
constexpr unsigned kLongRow = 512;

// What becomes of an entry: the new column alone, or (new row << 32 | column).
struct OutColumn {
  uint32_t* to;
  __device__ void put(uint64_t at, uint64_t, uint32_t col) const { to[at] = col; }
};
struct OutKey {
  uint64_t* to;
  __device__ void put(uint64_t at, uint64_t row, uint32_t col) const { to[at] = (row << 32) | col; }
};

// Row i of the copy is row list[i] of (off, adj) with its alive entries only
// (rem null: all of them), renumbered by newid, in noff[i] .. noff[i + 1] (an
// entry beyond that is dropped: a degree mismatch must not spill into the
// next row).  Warp per row of at most kLongRow entries.
template <class Out>
__global__ void __launch_bounds__(256) k_copy_rows(const uint32_t* __restrict__ list, uint64_t na,
                                                   const uint64_t* __restrict__ off, const uint32_t* __restrict__ adj,
                                                   const uint32_t* __restrict__ rem,
                                                   const uint32_t* __restrict__ newid,
                                                   const uint64_t* __restrict__ noff, Out out) {
  constexpr unsigned kPer = 4;
  const uint64_t warps = (uint64_t)gridDim.x * (blockDim.x >> 5);
  const unsigned lt = lanemask_lt();
  for (uint64_t i = (uint64_t)blockIdx.x * (blockDim.x >> 5) + warp_id(); i < na; i += warps) {
    const uint32_t v = list[i];
    const uint64_t b = off[v], e = off[v + 1];
    if (e - b > kLongRow) continue;  // k_copy_long_rows
    uint64_t pos = noff[i];
    const uint64_t end = noff[i + 1];
    for (uint64_t j0 = b; j0 < e; j0 += 32 * kPer) {
      const uint64_t j = j0 + lane_id();
      uint32_t w[kPer];
      bool keep[kPer];
#pragma unroll
      for (unsigned k = 0; k < kPer; ++k) w[k] = j + 32 * k < e ? adj[j + 32 * k] : 0u;
#pragma unroll
      for (unsigned k = 0; k < kPer; ++k) keep[k] = j + 32 * k < e && (rem == nullptr || rem[w[k]] == kAlive);
#pragma unroll
      for (unsigned k = 0; k < kPer; ++k) w[k] = keep[k] ? newid[w[k]] : 0u;
#pragma unroll
      for (unsigned k = 0; k < kPer; ++k) {
        const unsigned bal = __ballot_sync(kFull, keep[k]);
        const uint64_t p = pos + __popc(bal & lt);
        if (keep[k] && p < end) out.put(p, i, w[k]);
        pos += __popc(bal);
      }
    }
  }
}

// Indices of the list whose rows are longer than kLongRow.
struct LongListRow {
  const uint32_t* list;
  const uint64_t* off;
  __device__ bool keep(uint64_t i) const {
    const uint32_t v = list[i];
    return off[v + 1] - off[v] > kLongRow;
  }
  __device__ uint32_t value(uint64_t i) const { return (uint32_t)i; }
};

// The long rows (rows[0..nrows) are indices of the list): 256-entry windows
// dealt to every warp of the grid; a warp loads its window's 8 entries per
// lane, their alive flags and new ids before it uses any of them, and the
// kept entries go to the row's next free positions (a per-row cursor, one
// atomic per window).  Entry order within these rows is not kept.
template <class Out>
__global__ void __launch_bounds__(256) k_copy_long_rows(const uint32_t* __restrict__ rows, uint64_t nrows,
                                                        const uint32_t* __restrict__ list,
                                                        const uint64_t* __restrict__ off,
                                                        const uint32_t* __restrict__ adj,
                                                        const uint32_t* __restrict__ rem,
                                                        const uint32_t* __restrict__ newid,
                                                        const uint64_t* __restrict__ noff,
                                                        uint32_t* __restrict__ cursor, Out out) {
  __shared__ uint64_t woff[kBigBatch + 1];
  __shared__ uint64_t tmp[33];
  constexpr unsigned kPer = 8;
  const unsigned l = lane_id();
  deal_windows<32 * kPer>(
      nrows, [&](uint64_t x) { return list[rows[x]]; }, off, woff, tmp, [&](uint64_t x, uint64_t b, uint64_t e) {
        const uint32_t i = rows[x];
        const uint64_t j0 = b + l;
        uint32_t u[kPer];
#pragma unroll
        for (unsigned k = 0; k < kPer; ++k) u[k] = j0 + 32 * k < e ? adj[j0 + 32 * k] : 0u;
        bool keep[kPer];
#pragma unroll
        for (unsigned k = 0; k < kPer; ++k) keep[k] = j0 + 32 * k < e && (rem == nullptr || rem[u[k]] == kAlive);
#pragma unroll
        for (unsigned k = 0; k < kPer; ++k) u[k] = keep[k] ? newid[u[k]] : 0u;
        unsigned bal[kPer];
        uint32_t kept = 0;
#pragma unroll
        for (unsigned k = 0; k < kPer; ++k) {
          bal[k] = __ballot_sync(kFull, keep[k]);
          kept += __popc(bal[k]);
        }
        if (!kept) return;
        uint32_t at = 0;
        if (l == 0) at = atomicAdd(&cursor[x], kept);
        at = __shfl_sync(kFull, at, 0);
        const uint64_t row1 = noff[i + 1];
        uint64_t p0 = noff[i] + at;
#pragma unroll
        for (unsigned k = 0; k < kPer; ++k) {
          const uint64_t p = p0 + __popc(bal[k] & lanemask_lt());
          if (keep[k] && p < row1) out.put(p, i, u[k]);
          p0 += __popc(bal[k]);
        }
      });
}

// The copy of the rows of a list (max_deg: no row is longer).
template <class Out>
void copy_rows(Ctx* c, const uint32_t* list, uint64_t na, const uint64_t* off, const uint32_t* adj,
               const uint32_t* rem, const uint32_t* newid, const uint64_t* noff, uint32_t max_deg, Out out) {
  k_copy_rows<Out><<<grid_for(na * 32, 256, c->num_sms * 16), 256, 0, c->stream>>>(list, na, off, adj, rem, newid,
                                                                                   noff, out);
  KT_LAUNCHED(c);
  if (max_deg <= kLongRow) return;
  DBuf rows(c, (na ? na : 1) * sizeof(uint32_t));
  const uint64_t nlong = compact(c, na, LongListRow{list, off}, rows.as<uint32_t>());
  if (!nlong) return;
  DBuf cursor(c, nlong * sizeof(uint32_t));
  zero(c, cursor.get(), cursor.bytes());
  k_copy_long_rows<Out><<<c->num_sms * 8, 256, 0, c->stream>>>(rows.as<uint32_t>(), nlong, list, off, adj, rem, newid,
                                                               noff, cursor.as<uint32_t>(), out);
  KT_LAUNCHED(c);
}

}  // namespace kt
