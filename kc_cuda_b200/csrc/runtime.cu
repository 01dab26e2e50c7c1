// Context plumbing: device buffers charged to the HBM budget, small copies,
// and the CUDA error -> kt::Error conversion.
#include <algorithm>
#include <cstdio>
#include <cstring>
#include <mutex>
#include <set>
#include <utility>

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

// Whether a copy of `bytes` at host address p goes through the pinned slots:
// large, and to or from pageable memory, which the driver would stage with one
// thread (loading and solving 48 MB of records 5.6 -> 3.7 ms, 32 MB of supports
// counted and returned 6.8 -> 4.9 ms).
bool through_slots(Ctx* c, const void* p, size_t bytes) {
  if (bytes < (1 << 20)) return false;
  cudaPointerAttributes a;
  if (cudaPointerGetAttributes(&a, p) != cudaSuccess) {
    cudaGetLastError();
    return false;
  }
  if (a.type != cudaMemoryTypeUnregistered) return false;
  if (c->slots) return true;
  if (cudaHostAlloc(reinterpret_cast<void**>(&c->slots), kSlotBytes * kCopySlots, cudaHostAllocDefault) !=
      cudaSuccess) {
    cudaGetLastError();
    c->slots = nullptr;  // no pinned memory to be had: the driver's staging
    return false;
  }
  for (cudaEvent_t& e : c->slot_done)
    if (!e) KT_CUDA(cudaEventCreateWithFlags(&e, cudaEventDisableTiming));
  return true;
}

void parallel_memcpy(char* dst, const char* src, size_t n) {
  constexpr int kParts = 8;
#pragma omp parallel for schedule(static) num_threads(kParts)
  for (int t = 0; t < kParts; ++t) {
    const size_t a = n * t / kParts, b = n * (t + 1) / kParts;
    std::memcpy(dst + a, src + a, b - a);
  }
}

}  // namespace

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
  if (through_slots(c, dst, bytes)) {
    const size_t n = (bytes + kSlotBytes - 1) / kSlotBytes;
    auto size = [&](size_t i) { return std::min(kSlotBytes, bytes - i * kSlotBytes); };
    for (size_t i = 0; i < n + kCopySlots - 1; ++i) {
      if (i < n) {
        const int s = (int)(i % kCopySlots);
        KT_CUDA(cudaMemcpyAsync(c->slots + s * kSlotBytes, static_cast<const char*>(src) + i * kSlotBytes, size(i),
                                cudaMemcpyDeviceToHost, c->stream));
        KT_CUDA(cudaEventRecord(c->slot_done[s], c->stream));
      }
      if (i + 1 < kCopySlots) continue;  // keep kCopySlots - 1 copies ahead
      const size_t k = i + 1 - kCopySlots;
      const int s = (int)(k % kCopySlots);
      KT_CUDA(cudaEventSynchronize(c->slot_done[s]));
      parallel_memcpy(static_cast<char*>(dst) + k * kSlotBytes, c->slots + s * kSlotBytes, size(k));
    }
    return;
  }
  KT_CUDA(cudaMemcpyAsync(dst, src, bytes, cudaMemcpyDeviceToHost, c->stream));
  sync(c);
}

void copy_h2d(Ctx* c, void* dst, const void* src, size_t bytes) {
  if (!bytes) return;
  c->h2d_bytes += bytes;
  if (through_slots(c, src, bytes)) {
    for (size_t at = 0, i = 0; at < bytes; at += kSlotBytes, ++i) {
      const int s = (int)(i % kCopySlots);
      const size_t n = std::min(kSlotBytes, bytes - at);
      KT_CUDA(cudaEventSynchronize(c->slot_done[s]));
      parallel_memcpy(c->slots + s * kSlotBytes, static_cast<const char*>(src) + at, n);
      KT_CUDA(cudaMemcpyAsync(static_cast<char*>(dst) + at, c->slots + s * kSlotBytes, n, cudaMemcpyHostToDevice,
                              c->stream));
      KT_CUDA(cudaEventRecord(c->slot_done[s], c->stream));
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
