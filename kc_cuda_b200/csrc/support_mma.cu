// Supports of dense working graphs on the tensor cores.
//
// The support of an edge (u, v) is entry (u, v) of the square of the adjacency
// matrix.  The rows' bitsets are expanded to bytes (0 or 1) and multiplied as
// 8-bit integers with 32-bit sums, so the counts are exact; only the tiles on
// and above the diagonal are formed, and an edge's count is taken from its tile
// as it leaves the accumulator.
//
// A popcount of two rows reads W words per edge from L2 and is bound by that:
// 3.07 G words, 12.3 GB, in 1.52 ms for the 9,022-vertex maximum core of an
// R-MAT scale 22 graph (10.5M edges).  A tile of 256 x 256 reads 512 rows for
// 65,536 products whatever its edges are, so its traffic and its time follow n^3
// alone, and product_pays has the line between the two.  That core takes 0.31 ms
// (0.27 the product: 666 tiles, 0.75 P operations, 2.8 P/s; 3.4 at 13,000
// vertices, 4.1 at 36,000), the 9,109 vertices and 10.6M edges of the search 0.34
// instead of 2.62 (capped popcounts), a union of 63,796 vertices, 18.8M edges in
// graphs of up to 6,178 vertices 0.82 instead of 3.80 ms.
//
// One block per SM keeps a queue of kStages stages, each 128 columns (128
// bytes) of 256 rows of either side, brought in by TMA with 128-byte swizzling.
// Warp 0 issues the copies, warp 1 the tcgen05.mma (two accumulators of 128 x
// 256, all 512 columns of tensor memory: a tile of 128 x 256 would read 1.5
// times the bytes per product), the other eight warps take the counts out, each
// thread a row of 256 columns.
#include <cuda.h>

#include <algorithm>
#include <vector>

#include "dense.cuh"
#include "stages.h"
#include "subgraph.h"
#include "support_mma.h"
#include "teams.h"

namespace kt {
namespace {

constexpr uint32_t kTile = 256;   // rows and columns of a tile
constexpr uint32_t kDepth = 128;  // columns of a stage
constexpr uint32_t kStages = 3;
constexpr uint32_t kHalfBytes = 128 * kDepth;       // one operand of a tcgen05.mma with 128 rows
constexpr uint32_t kSideBytes = 2 * kHalfBytes;     // 256 rows
constexpr uint32_t kStageBytes = 2 * kSideBytes;    // rows of u and rows of v
constexpr unsigned kMmaThreads = 320;
constexpr unsigned kOutWarps = 8;
constexpr size_t kMmaSmem = kStages * kStageBytes + 1024;  // (stages start on 1024 bytes)
constexpr uint32_t kTmemCols = 512;
constexpr unsigned long long kDrainNs = 2000000000ULL;  // bound on a block's last waits, for its own copies and products

// Instruction descriptor of tcgen05.mma kind::i8: unsigned bytes, 32-bit sums,
// both sides with consecutive columns in a row, 128 x 256.
constexpr uint32_t kInstr = (2u << 4) | ((256u >> 3) << 17) | ((128u >> 4) << 24);

__device__ __forceinline__ uint32_t smem_addr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

// Shared-memory descriptor of rows of 128 bytes, 128-byte swizzle (8 rows are
// 1024 bytes apart from the next 8).
__device__ __forceinline__ uint64_t rows_desc(uint32_t addr) {
  return (uint64_t)((addr & 0x3ffff) >> 4) | (1ull << 16) | ((1024ull >> 4) << 32) | (1ull << 46) | (2ull << 61);
}

// Waits for the phase of `parity`, at most `timeout_ns` and not after another
// role of the block has given up; false then, with *quit set and kDevErrWait
// flagged.
__device__ __forceinline__ bool wait_phase(uint32_t bar, uint32_t parity, unsigned long long timeout_ns,
                                           volatile uint32_t* quit, uint32_t* err) {
  unsigned long long t0 = 0;
  while (true) {
    uint32_t done;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}"
        : "=r"(done)
        : "r"(bar), "r"(parity)
        : "memory");
    if (done) return true;
    const unsigned long long now = globaltimer_ns();
    if (!t0) t0 = now;
    if (*quit || now - t0 >= timeout_ns) {
      *quit = 1;
      atomicOr(err, kDevErrWait);
      return false;
    }
  }
}

__device__ __forceinline__ void bar_init(uint32_t bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}

__device__ __forceinline__ void load_rows(uint32_t dst, const CUtensorMap* map, uint32_t x, uint32_t y, uint32_t bar) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(
          dst),
      "l"(map), "r"(x), "r"(y), "r"(bar)
      : "memory");
}

__device__ __forceinline__ void mma_i8(uint32_t acc, uint64_t a, uint64_t b, bool add) {
  asm volatile(
      "{\n .reg .pred p;\n setp.ne.u32 p, %4, 0;\n tcgen05.mma.cta_group::1.kind::i8 [%0], %1, %2, %3, p;\n}" ::"r"(acc),
      "l"(a), "l"(b), "r"(kInstr), "r"((uint32_t)add)
      : "memory");
}

__device__ __forceinline__ void mma_arrive(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}

__device__ __forceinline__ void acc_load32(uint32_t at, uint32_t* r) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
      "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];\n"
      "tcgen05.wait::ld.sync.aligned;"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]),
        "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]),
        "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(at)
      : "memory");
}

// One graph of the union (or all of the working graph): vertices v0 .. v0 + n,
// rows of W words, its tiles numbered from tile0.
struct MmaBlock {
  uint64_t words;   // its first word in the bitsets
  uint64_t bytes;   // its first byte in the expanded rows
  uint64_t tile0;
  uint32_t v0, n, W, side;  // side: tiles per row of tiles
};

struct MmaArgs {
  const CUtensorMap* maps;  // one per block
  const MmaBlock* blocks;
  uint32_t nblocks;
  uint64_t tiles;
  DenseRows R;
  const uint64_t* off;
  const uint64_t* up;
  const uint32_t* eid;
  uint32_t* sup;
  uint32_t* err;
  unsigned long long timeout_ns;
};

constexpr uint32_t kSquare = 12;

// Tile t: its block, and its place (i, j) with i <= j.
__device__ __forceinline__ uint32_t find_tile(const MmaArgs& A, uint64_t t, uint32_t& i, uint32_t& j) {
  uint32_t lo = 0, hi = A.nblocks;
  while (hi - lo > 1) {
    const uint32_t mid = (lo + hi) >> 1;
    if (A.blocks[mid].tile0 <= t)
      lo = mid;
    else
      hi = mid;
  }
  // Squares of kSquare x kSquare tiles one after another: the tiles in flight
  // share 2 * kSquare row stretches, where a row of tiles would read every row of
  // the matrix from memory again once it is beyond L2.
  uint64_t x = t - A.blocks[lo].tile0;
  const uint32_t side = A.blocks[lo].side;
  uint32_t i0 = 0, j0 = 0, rows = min(kSquare, side), cols = rows;
  while (true) {
    const uint32_t n = i0 == j0 ? rows * (rows + 1) / 2 : rows * cols;
    if (x < n) break;
    x -= n;
    j0 += kSquare;
    if (j0 >= side) {
      i0 += kSquare;
      j0 = i0;
      rows = min(kSquare, side - i0);
    }
    cols = min(kSquare, side - j0);
  }
  if (i0 != j0) {
    i = i0 + (uint32_t)x % rows;
    j = j0 + (uint32_t)x / rows;
  } else {
    uint32_t y = 0;
    while (x >= rows - y) x -= rows - y++;
    i = i0 + y;
    j = i + (uint32_t)x;
  }
  return lo;
}

// 16 bits of a row -> 16 bytes.
__global__ void __launch_bounds__(256) k_expand_rows(const uint32_t* __restrict__ bits,
                                                     const MmaBlock* __restrict__ blocks, uint8_t* __restrict__ out) {
  const MmaBlock B = blocks[blockIdx.y];
  const uint64_t halves = 2ull * B.n * B.W;
  const uint16_t* src = reinterpret_cast<const uint16_t*>(bits + B.words);
  uint4* dst = reinterpret_cast<uint4*>(out + B.bytes);
  for (uint64_t h = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; h < halves; h += (uint64_t)gridDim.x * blockDim.x) {
    const uint32_t x = src[h];
    uint32_t w[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) w[q] = (((x >> (4 * q)) & 15u) * 0x00204081u) & 0x01010101u;
    dst[h] = make_uint4(w[0], w[1], w[2], w[3]);
  }
}

__global__ void __launch_bounds__(kMmaThreads, 1) k_support_mma(MmaArgs A) {
  extern __shared__ uint8_t raw[];
  __shared__ uint64_t bars[2 * kStages + 3];
  __shared__ uint32_t tmem;
  __shared__ volatile uint32_t quit;
  const uint32_t stage0 = (smem_addr(raw) + 1023) & ~1023u;
  const unsigned warp = warp_id(), lane = lane_id();
  const uint32_t full = smem_addr(&bars[0]), empty = smem_addr(&bars[kStages]);
  const uint32_t acc_full = smem_addr(&bars[2 * kStages]), acc_empty = acc_full + 8, drain = acc_full + 16;
  if (threadIdx.x == 0) {
    for (uint32_t s = 0; s < kStages; ++s) {
      bar_init(full + 8 * s, 1);
      bar_init(empty + 8 * s, 1);
    }
    bar_init(acc_full, 1);
    bar_init(acc_empty, kOutWarps);
    bar_init(drain, 1);
    quit = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_addr(&tmem)),
                 "r"(kTmemCols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t acc = tmem;

  if (warp == 0) {
    if (lane == 0) {
      uint32_t it = 0;
      bool ok = true;
      for (uint64_t t = blockIdx.x; t < A.tiles && ok; t += gridDim.x) {
        uint32_t i, j;
        const uint32_t b = find_tile(A, t, i, j);
        const uint32_t steps = A.blocks[b].W / 4;
        const CUtensorMap* map = A.maps + b;
        asm volatile("fence.proxy.tensormap::generic.acquire.sys [%0], 128;" ::"l"(map) : "memory");
        for (uint32_t k = 0; k < steps; ++k, ++it) {
          const uint32_t s = it % kStages;
          ok = wait_phase(empty + 8 * s, ((it / kStages) & 1) ^ 1, A.timeout_ns, &quit, A.err);
          if (!ok) break;
          const uint32_t bar = full + 8 * s, at = stage0 + s * kStageBytes;
          asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(kStageBytes) : "memory");
          load_rows(at, map, k * kDepth, i * kTile, bar);
          load_rows(at + kSideBytes, map, k * kDepth, j * kTile, bar);
        }
      }
      // The copies in flight end before the block does: also where all of them
      // were issued, since the products may have given up on the last ones.
      for (uint32_t x = it > kStages ? it - kStages : 0; x < it; ++x) {
        volatile uint32_t none = 0;
        wait_phase(full + 8 * (x % kStages), (x / kStages) & 1, kDrainNs, &none, A.err);
      }
    }
  } else if (warp == 1) {
    if (lane == 0) {
      uint32_t it = 0, nt = 0;
      bool ok = true;
      for (uint64_t t = blockIdx.x; t < A.tiles && ok; t += gridDim.x, ++nt) {
        uint32_t i, j;
        const uint32_t b = find_tile(A, t, i, j);
        const uint32_t steps = A.blocks[b].W / 4;
        ok = wait_phase(acc_empty, (nt & 1) ^ 1, A.timeout_ns, &quit, A.err);
        if (!ok) break;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        for (uint32_t k = 0; k < steps; ++k, ++it) {
          const uint32_t s = it % kStages;
          ok = wait_phase(full + 8 * s, (it / kStages) & 1, A.timeout_ns, &quit, A.err);
          if (!ok) break;
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          const uint32_t at = stage0 + s * kStageBytes;
          const uint64_t u = rows_desc(at), v = rows_desc(at + kSideBytes);
#pragma unroll
          for (uint32_t q = 0; q < kDepth / 32; ++q) {  // 32 columns a time: 2 units of 16 bytes
            mma_i8(acc, u + 2 * q, v + 2 * q, k || q);
            mma_i8(acc + kTile, u + (kHalfBytes >> 4) + 2 * q, v + 2 * q, k || q);
          }
          mma_arrive(empty + 8 * s);
        }
        if (ok) mma_arrive(acc_full);
      }
      // So do the products, before the tensor memory is given back.
      mma_arrive(drain);
      volatile uint32_t none = 0;
      wait_phase(drain, 0, kDrainNs, &none, A.err);
    }
  } else {
    const unsigned half = (warp - 2) >> 2, quad = warp & 3;  // a warp reaches the 32 lanes of its place in four
    const uint32_t from = acc + half * kTile + ((quad * 32u) << 16);
    uint32_t nt = 0;
    for (uint64_t t = blockIdx.x; t < A.tiles; t += gridDim.x, ++nt) {
      uint32_t i, j;
      const MmaBlock& B = A.blocks[find_tile(A, t, i, j)];
      const uint32_t row = i * kTile + half * 128 + quad * 32 + lane;  // within the block
      const bool real = row < B.n;
      // The row's bits in these columns and the id of the first edge there,
      // read while the products run.
      uint32_t bits[kTile / 32] = {};
      uint32_t id = 0;
      if (real && j * kTile + kTile > row) {
        const uint32_t u = B.v0 + row;
        const uint64_t at = B.words + (uint64_t)row * B.W + j * (kTile / 32);
        *reinterpret_cast<uint4*>(bits) = *reinterpret_cast<const uint4*>(A.R.sbits + at);
        if (j * (kTile / 32) + 4 < B.W)
          *reinterpret_cast<uint4*>(bits + 4) = *reinterpret_cast<const uint4*>(A.R.sbits + at + 4);
        const uint64_t pu = A.up[u], b = A.off[u];
        if (pu < A.off[u + 1]) id = A.eid[pu] + A.R.spre[at] - (uint32_t)(pu - b);
      }
      const bool ok = __all_sync(kFull, wait_phase(acc_full, nt & 1, A.timeout_ns, &quit, A.err));
      if (!ok) break;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
      for (uint32_t w = 0; w < kTile / 32; ++w) {
        const uint32_t col = j * kTile + 32 * w;  // columns up to the row itself are the lower neighbours
        const uint32_t below = row >= col + 31 ? ~0u : row < col ? 0u : (2u << (row - col)) - 1u;
        uint32_t e = id + __popc(bits[w] & below);
        const uint32_t m = bits[w] & ~below;
        id += __popc(bits[w]);
        if (!__any_sync(kFull, m)) continue;
        uint32_t r[32];
        acc_load32(from + 32 * w, r);
        // (Gathering a row's counts in shared memory for longer stores gave 4 %
        // on dense rows and took 10 % on sparse ones.)
#pragma unroll
        for (int q = 0; q < 32; ++q)
          if ((m >> q) & 1u) A.sup[e++] = r[q];
      }
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      __syncwarp();
      if (lane == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(acc_empty) : "memory");
    }
  }
  __syncwarp();
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == 1) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(acc), "r"(kTmemCols));
  }
}

using EncodeTiled = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                 const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                 CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiled encode_tiled() {
  static const EncodeTiled fn = [] {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult r;
    if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault, &r) != cudaSuccess ||
        r != cudaDriverEntryPointSuccess) {
      cudaGetLastError();
      p = nullptr;
    }
    return reinterpret_cast<EncodeTiled>(p);
  }();
  return fn;
}

// Rows of W words, one byte per bit, at `base`.
CUtensorMap rows_map(void* base, uint32_t n, uint32_t W) {
  CUtensorMap map;
  const cuuint64_t dims[2] = {(cuuint64_t)W * 32, n}, strides[1] = {(cuuint64_t)W * 32};
  const cuuint32_t box[2] = {kDepth, kTile}, step[2] = {1, 1};
  const CUresult r = encode_tiled()(&map, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, base, dims, strides, box, step,
                                    CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                                    CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) throw Error(KT_ERR_CUDA, "support: tensor map refused");
  return map;
}

// Whether the product of a graph's rows takes less time than a popcount of W
// words per edge, both with the whole GPU working on graphs like it.  A tile
// measures 0.55-0.6 us for 128 columns (the rate of the tensor cores) and up to 18
// beyond that for its counts' way out, the launches and the byte rows about 20 in
// all.  Popcounts of rows of up to kShortRow words go at 1.1 G words a
// millisecond; of longer ones they take a time per edge up to some 600 words and
// 3.5 G words a millisecond beyond, capped ones more time per edge but up to 5.5
// G words for those they abandon.  So the line lies between 4 and 8 % of a
// graph's pairs (exact counts at 12 %: 9,100 vertices 0.27 ms as products, 0.72
// as popcounts; 36,000 vertices 11.5 and 23.7 ms; capped counts of 92M edges on
// 55,455 vertices, 6 %: about 42 and 30).
bool product_pays(uint64_t m, uint32_t W, uint64_t tiles, unsigned sms, bool alone, bool capped) {
  const double rounds = alone ? (double)((tiles + sms - 1) / sms) : (double)tiles / sms;
  const double product_us = (alone ? 20.0 : 0.0) + rounds * (18.0 + 0.57 * (W / 4));
  const double words_per_us = W <= kShortRow ? 1.1e6
                              : capped       ? std::min(4.1e3 * W, 5.5e6)
                                             : std::min(5.5e3 * W, 3.5e6);
  return product_us < (double)m * W / words_per_us;
}

}  // namespace

bool support_products(Ctx* c, const Sub& s, uint32_t* sup, bool capped, std::vector<uint8_t>& counted,
                      uint64_t* words) {
  *words = 0;
  // (Not where rounds are host-stepped: a block here takes an SM's shared memory,
  // so a lane that runs beside another's cooperative grids would wait for them.)
  if (!s.W || !s.spre.get() || !c->opt.persistent || !encode_tiled()) return false;
  std::vector<MmaBlock> blocks;
  uint64_t row_bytes = 0;
  auto add = [&](uint64_t first_word, uint32_t v0, uint32_t n, uint32_t W) {
    blocks.push_back(MmaBlock{first_word, 0, 0, v0, n, W, (n + kTile - 1) / kTile});
    row_bytes += (uint64_t)n * W * 32;
  };
  auto tiles_of = [](uint32_t n) {
    const uint64_t side = (n + kTile - 1) / kTile;
    return side * (side + 1) / 2;
  };
  if (!s.roff.get()) {
    if (!product_pays(s.m, s.W, tiles_of(s.n), c->num_sms, true, capped)) return false;
    add(0, 0, s.n, s.W);
  } else {
    // (Its launches have to pay as well: 2e6 words take a microsecond.)
    constexpr double kLeastWords = 100e6;
    if ((double)s.m * s.W < kLeastWords) return false;
    const uint32_t G = (uint32_t)s.group_n.size();
    std::vector<uint64_t> starts(G + 1, 0);
    for (uint32_t g = 0; g < G; ++g) starts[g + 1] = starts[g] + s.group_n[g];
    const std::vector<uint64_t> at = gather_offsets(c, s.off.as<uint64_t>(), starts);
    counted.assign(G, 0);
    uint64_t word = 0;
    double gain = 0;
    for (uint32_t g = 0; g < G; ++g) {
      const uint32_t n = s.group_n[g], W = ((n + 31) / 32 + 3) & ~3u;
      const uint64_t m = (at[g + 1] - at[g]) / 2;
      if (n && blocks.size() < 65535 && product_pays(m, W, tiles_of(n), c->num_sms, false, capped)) {
        add(word, (uint32_t)starts[g], n, W);
        counted[g] = 1;
        gain += (double)m * W;
      }
      word += (uint64_t)n * W;
    }
    if (gain < kLeastWords) return false;
  }
  if (c->budget && c->in_use + row_bytes + blocks.size() * 256 + 4096 > c->budget) return false;
  DBuf rows;
  if (!rows.try_alloc(c, row_bytes)) return false;  // the popcounts need no room
  // The longest first: a block of the grid takes every 148th tile.
  std::sort(blocks.begin(), blocks.end(), [](const MmaBlock& a, const MmaBlock& b) { return a.W > b.W; });
  std::vector<CUtensorMap> maps;
  uint64_t tiles = 0, at = 0, most = 0;
  for (MmaBlock& B : blocks) {
    B.bytes = at;
    B.tile0 = tiles;
    maps.push_back(rows_map(rows.as<uint8_t>() + at, B.n, B.W));
    at += (uint64_t)B.n * B.W * 32;
    tiles += tiles_of(B.n);
    most = std::max<uint64_t>(most, 2ull * B.n * B.W);
    *words += tiles_of(B.n) * (B.W / 4) * (kStageBytes / 4);
  }
  DBuf dmaps(c, maps.size() * sizeof(CUtensorMap)), dblocks(c, blocks.size() * sizeof(MmaBlock));
  copy_h2d(c, dmaps.get(), maps.data(), maps.size() * sizeof(CUtensorMap));
  copy_h2d(c, dblocks.get(), blocks.data(), blocks.size() * sizeof(MmaBlock));
  const unsigned per = std::max<unsigned>(1, c->num_sms * 16 / (unsigned)blocks.size());
  k_expand_rows<<<dim3(grid_for(most, 256, per), (unsigned)blocks.size()), 256, 0, c->stream>>>(
      s.bits.as<uint32_t>(), dblocks.as<MmaBlock>(), rows.as<uint8_t>());
  KT_LAUNCHED(c);
  MmaArgs A;
  A.maps = dmaps.as<CUtensorMap>();
  A.blocks = dblocks.as<MmaBlock>();
  A.nblocks = (uint32_t)blocks.size();
  A.tiles = tiles;
  A.R = dense_rows(s);
  A.off = s.off.as<uint64_t>();
  A.up = s.up.as<uint64_t>();
  A.eid = s.eid.as<uint32_t>();
  A.sup = sup;
  A.err = &dev_words(c)->err;
  A.timeout_ns = (unsigned long long)c->opt.timeout_ms * 1000000ULL;
  allow_max_dynamic_smem((const void*)k_support_mma);
  k_support_mma<<<(unsigned)std::min<uint64_t>(tiles, c->num_sms), kMmaThreads, kMmaSmem, c->stream>>>(A);
  KT_LAUNCHED(c);
  return true;
}

}  // namespace kt
