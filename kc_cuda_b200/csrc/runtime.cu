// Context plumbing: device buffers charged to the HBM budget, small copies,
// and the CUDA error -> kt::Error conversion.
#include <omp.h>

#include <algorithm>
#include <cstdio>
#include <cstring>
#include <map>
#include <mutex>
#include <new>
#include <set>
#include <utility>
#include <vector>

#include "kt_internal.h"

namespace kt {

void throw_cuda(cudaError_t e, const char* what, const char* file, int line) {
  char buf[512];
  std::snprintf(buf, sizeof(buf), "%s: %s (%s:%d)", what, cudaGetErrorString(e), file, line);
  cudaGetLastError();  // clear a sticky launch error where possible
  kt_status s = (e == cudaErrorMemoryAllocation) ? KT_ERR_NOMEM : KT_ERR_CUDA;
  throw Error(s, buf);
}

void DBuf::alloc(Ctx* c, size_t bytes) {
  ctx_ = c;
  bytes_ = 0;
  ptr_ = nullptr;
  if (bytes == 0) bytes = 16;
  bytes = (bytes + 255) & ~size_t(255);
  if (c->budget && c->in_use + bytes > c->budget) {
    char buf[256];
    std::snprintf(buf, sizeof(buf), "HBM budget exceeded: %zu bytes requested, %llu of %llu in use", bytes,
                  (unsigned long long)c->in_use, (unsigned long long)c->budget);
    throw Error(KT_ERR_NOMEM, buf);
  }
  cudaError_t e = cudaMallocAsync(&ptr_, bytes, c->stream);
  if (e != cudaSuccess) {
    ptr_ = nullptr;
    throw_cuda(e, "cudaMallocAsync", __FILE__, __LINE__);
  }
  bytes_ = bytes;
  c->in_use += bytes;
  if (c->in_use > c->peak) c->peak = c->in_use;
}

void DBuf::release() {
  if (ptr_ && ctx_) {
    cudaFreeAsync(ptr_, ctx_->stream);
    ctx_->in_use -= bytes_;
  }
  ptr_ = nullptr;
  bytes_ = 0;
  ctx_ = nullptr;
}

void allow_max_dynamic_smem(const void* func) {
  static std::mutex mu;
  static std::set<std::pair<int, const void*>> done;
  int dev = 0;
  KT_CUDA(cudaGetDevice(&dev));
  std::lock_guard<std::mutex> lk(mu);
  if (done.count({dev, func})) return;
  int optin = 0;
  KT_CUDA(cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev));
  cudaFuncAttributes fa;
  KT_CUDA(cudaFuncGetAttributes(&fa, func));
  KT_CUDA(cudaFuncSetAttribute(func, cudaFuncAttributeMaxDynamicSharedMemorySize,
                               optin - (int)fa.sharedSizeBytes));
  done.insert({dev, func});
}

void sync(Ctx* c) { KT_CUDA(cudaStreamSynchronize(c->stream)); }

namespace {

constexpr size_t kSlotBytes = 4 << 20;
constexpr int kCopySlots = 4;

// Pinned slots for large copies from and to pageable memory, which the driver
// would stage with one thread (48 MB to the device 2.9 -> 1.1 ms, back 2.6 ->
// 1.0; slots of 1 MB 1.8, of 256 KB 1.9).  Pinning these 16 MB takes 15 ms, so
// they are made once the copies of a device have lost a part of that to the
// driver's staging (kSlotsAfter bytes, about 5 ms), and then serve all contexts
// there: made by a context's first large copy, they cost a program of one call, and
// each lane of a new server, more than all that they saved it.
struct CopySlots {
  int device;
  char* bytes = nullptr;
  cudaEvent_t done[kCopySlots] = {};  // each slot's last copy
  ~CopySlots() {
    for (cudaEvent_t e : done)
      if (e) {
        cudaEventSynchronize(e);
        cudaEventDestroy(e);
      }
    if (bytes) cudaFreeHost(bytes);
    cudaGetLastError();
  }
};
constexpr uint64_t kSlotsAfter = 128ull << 20;
constexpr int kMostSlots = 4;  // sets on a device: copies at once that have slots

struct SlotPool {
  std::mutex mu;
  struct Device {
    std::vector<CopySlots*> idle;
    int made = 0;
    uint64_t staged = 0;  // bytes left to the driver since the last set was made
  };
  std::map<int, Device> devices;
};
SlotPool& slot_pool() {
  static SlotPool* p = new SlotPool;  // (never destroyed: contexts may outlive static objects)
  return *p;
}

// A set of slots for one copy, where it is large and to or from pageable memory
// and a set is idle or may be made.
class SlotLease {
 public:
  SlotLease(Ctx* c, const void* p, size_t bytes) {
    if (bytes < (1 << 20)) return;
    cudaPointerAttributes a;
    if (cudaPointerGetAttributes(&a, p) != cudaSuccess) {
      cudaGetLastError();
      return;
    }
    if (a.type != cudaMemoryTypeUnregistered) return;
    SlotPool& pool = slot_pool();
    {
      std::lock_guard<std::mutex> lk(pool.mu);
      SlotPool::Device& d = pool.devices[c->device];
      if (!d.idle.empty()) {
        s_ = d.idle.back();
        d.idle.pop_back();
        return;
      }
      d.staged += bytes;
      if (d.made == kMostSlots || d.staged < kSlotsAfter) return;
      d.idle.reserve(kMostSlots);  // giving a set back does not allocate
      d.staged = 0;
      ++d.made;
    }
    CopySlots* s = new (std::nothrow) CopySlots{c->device};
    bool ok = s && cudaHostAlloc(reinterpret_cast<void**>(&s->bytes), kSlotBytes * kCopySlots,
                                 cudaHostAllocPortable) == cudaSuccess;
    for (int i = 0; ok && i < kCopySlots; ++i)
      ok = cudaEventCreateWithFlags(&s->done[i], cudaEventDisableTiming) == cudaSuccess;
    if (ok) {
      s_ = s;
      return;
    }
    cudaGetLastError();  // no pinned memory to be had: the driver's staging
    delete s;
    std::lock_guard<std::mutex> lk(pool.mu);
    --pool.devices[c->device].made;
  }
  ~SlotLease() {
    if (!s_) return;
    SlotPool& pool = slot_pool();
    std::lock_guard<std::mutex> lk(pool.mu);
    pool.devices[s_->device].idle.push_back(s_);
  }
  SlotLease(const SlotLease&) = delete;
  SlotLease& operator=(const SlotLease&) = delete;
  explicit operator bool() const { return s_ != nullptr; }
  char* slot(size_t i) const { return s_->bytes + i % kCopySlots * kSlotBytes; }
  cudaEvent_t done(size_t i) const { return s_->done[i % kCopySlots]; }

 private:
  CopySlots* s_ = nullptr;
};

void parallel_memcpy(char* dst, const char* src, size_t n) {
  constexpr int kParts = 8;
#pragma omp parallel for schedule(static) num_threads(copy_threads())
  for (int t = 0; t < kParts; ++t) {
    const size_t a = n * t / kParts, b = n * (t + 1) / kParts;
    std::memcpy(dst + a, src + a, b - a);
  }
}

}  // namespace

int copy_threads() {
  static const int n = std::max(1, std::min(8, omp_get_num_procs()));
  return n;
}

void release_copy_slots(int device) {
  std::vector<CopySlots*> sets;
  {
    SlotPool& pool = slot_pool();
    std::lock_guard<std::mutex> lk(pool.mu);
    SlotPool::Device& d = pool.devices[device];
    sets.swap(d.idle);
    d.made -= (int)sets.size();
    d.staged = 0;
  }
  for (CopySlots* s : sets) delete s;
}

void copy_d2h(Ctx* c, void* dst, const void* src, size_t bytes) {
  if (!bytes) return;
  c->d2h_bytes += bytes;
  if (bytes <= kPinnedBytes) {
    // Small results through the context's pinned words: a copy to pageable
    // memory is staged by the driver.
    KT_CUDA(cudaMemcpyAsync(c->pinned, src, bytes, cudaMemcpyDeviceToHost, c->stream));
    sync(c);
    std::memcpy(dst, c->pinned, bytes);
    return;
  }
  if (SlotLease slots{c, dst, bytes}) {
    const size_t n = (bytes + kSlotBytes - 1) / kSlotBytes;
    auto size = [&](size_t i) { return std::min(kSlotBytes, bytes - i * kSlotBytes); };
    for (size_t i = 0; i < n + kCopySlots - 1; ++i) {
      if (i < n) {
        // (A copy that had the slots before may still read them, on another stream.)
        if (i < kCopySlots) KT_CUDA(cudaEventSynchronize(slots.done(i)));
        KT_CUDA(cudaMemcpyAsync(slots.slot(i), static_cast<const char*>(src) + i * kSlotBytes, size(i),
                                cudaMemcpyDeviceToHost, c->stream));
        KT_CUDA(cudaEventRecord(slots.done(i), c->stream));
      }
      if (i + 1 < kCopySlots) continue;  // keep kCopySlots - 1 copies ahead
      const size_t k = i + 1 - kCopySlots;
      KT_CUDA(cudaEventSynchronize(slots.done(k)));
      parallel_memcpy(static_cast<char*>(dst) + k * kSlotBytes, slots.slot(k), size(k));
    }
    return;
  }
  KT_CUDA(cudaMemcpyAsync(dst, src, bytes, cudaMemcpyDeviceToHost, c->stream));
  sync(c);
}

void copy_h2d(Ctx* c, void* dst, const void* src, size_t bytes) {
  if (!bytes) return;
  c->h2d_bytes += bytes;
  if (SlotLease slots{c, src, bytes}) {
    for (size_t at = 0, i = 0; at < bytes; at += kSlotBytes, ++i) {
      const size_t n = std::min(kSlotBytes, bytes - at);
      KT_CUDA(cudaEventSynchronize(slots.done(i)));
      parallel_memcpy(slots.slot(i), static_cast<const char*>(src) + at, n);
      KT_CUDA(cudaMemcpyAsync(static_cast<char*>(dst) + at, slots.slot(i), n, cudaMemcpyHostToDevice, c->stream));
      KT_CUDA(cudaEventRecord(slots.done(i), c->stream));
    }
    return;
  }
  KT_CUDA(cudaMemcpyAsync(dst, src, bytes, cudaMemcpyHostToDevice, c->stream));
}

void zero(Ctx* c, void* dptr, size_t bytes) {
  if (!bytes) return;
  KT_CUDA(cudaMemsetAsync(dptr, 0, bytes, c->stream));
}

cudaEvent_t EventTimer::get() {
  if (used == pool.size()) {
    cudaEvent_t e;
    KT_CUDA(cudaEventCreate(&e));
    pool.push_back(e);
  }
  return pool[used++];
}

void EventTimer::begin(cudaStream_t s, double* acc, cudaEvent_t* out_a) {
  (void)acc;
  *out_a = get();
  KT_CUDA(cudaEventRecord(*out_a, s));
}

void EventTimer::end(cudaStream_t s, cudaEvent_t a, double* acc) {
  cudaEvent_t b = get();
  KT_CUDA(cudaEventRecord(b, s));
  open.push_back({a, b, acc});
}

void EventTimer::resolve() {
  for (const Span& sp : open) {
    KT_CUDA(cudaEventSynchronize(sp.b));
    float ms = 0;
    KT_CUDA(cudaEventElapsedTime(&ms, sp.a, sp.b));
    *sp.acc += ms;
  }
  open.clear();
  used = 0;
}

EventTimer::~EventTimer() {
  for (cudaEvent_t e : pool) cudaEventDestroy(e);
}

}  // namespace kt
