// Batched solving (batch.cu).
#pragma once
#include <memory>
#include <vector>

#include "stages.h"

namespace kt {

// Vectors whose elements are written before they are read: resize() leaves
// them uninitialised, so their pages are first touched by who fills them.
template <class T>
struct UninitAllocator : std::allocator<T> {
  template <class U>
  struct rebind {
    using other = UninitAllocator<U>;
  };
  template <class U>
  void construct(U* p) noexcept {
    ::new (static_cast<void*>(p)) U;
  }
  template <class U, class A, class... R>
  void construct(U* p, A&& a, R&&... r) {
    ::new (static_cast<void*>(p)) U(std::forward<A>(a), std::forward<R>(r)...);
  }
};
using Records = std::vector<uint64_t, UninitAllocator<uint64_t>>;

// One graph of a batch: generated on the device from a mix spec, or host
// records x << 32 | y.
struct BatchItem {
  bool generated = false;
  uint32_t kind = 0, scale = 0;
  uint64_t n = 0;      // vertex id range
  uint64_t draws = 0;  // generated draws
  uint64_t seed = 0;
  uint64_t nkeys = 0;  // draws + extra
  Records extra;       // clique keys (generated) or the records (host)
  uint32_t kmax = 0;
  uint64_t count = 0;
  void from_mix(uint64_t index, uint64_t base_seed);
  void from_pairs(const uint64_t* xy, uint64_t count);
};

struct BatchRun {
  uint32_t waves = 0;
};

void solve_wave(Ctx* c, const std::vector<BatchItem*>& items);
void run_batch(Ctx* c, std::vector<BatchItem>& items, BatchRun& out);
// Graph `index` of the batched mix, generated on the device.
void load_mix_graph(Ctx* c, uint64_t index, uint64_t base_seed, Graph& g);

}  // namespace kt
