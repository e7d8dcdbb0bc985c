// Internal: errors, blocking uploads and the device arena (host code only).
#pragma once

#include <algorithm>
#include <stdexcept>
#include <string>
#include <vector>

#include <cuda_runtime_api.h>

#include "../../include/anb.h"

namespace anb {

struct AnbError : std::runtime_error {
  int code;
  AnbError(int c, const std::string& m) : std::runtime_error(m), code(c) {}
};

#define CK(call)                                                                                          \
  do {                                                                                                    \
    cudaError_t e_ = (call);                                                                              \
    if (e_ != cudaSuccess)                                                                                \
      throw AnbError(ANB_ERR_CUDA, std::string("CUDA error ") + cudaGetErrorString(e_) + " at " #call);   \
  } while (0)

// Copies pageable host memory to the device and waits until it is there.  cudaMemcpy alone may return while
// its last staged part is still on its way, and the contexts' non-blocking streams are not ordered after it.
inline void upload_now(void* dst, const void* src, size_t bytes) {
  if (bytes == 0) return;
  CK(cudaMemcpy(dst, src, bytes, cudaMemcpyHostToDevice));
  CK(cudaStreamSynchronize(cudaStreamLegacy));
}

// An allocation that the device has no room for.
struct NoDeviceMemory : AnbError {
  explicit NoDeviceMemory(size_t bytes)
      : AnbError(ANB_ERR_CUDA, "CUDA error out of memory for " + std::to_string(bytes) + " bytes") {}
};

// Device allocations owned by a context, cut from slabs and given back together.  A cudaMalloc takes 0.33 ms
// and a cudaFree 0.27 ms whatever the size up to 64 MB, and a hierarchy makes about 60: requests below
// kOwnSlab share slabs of at most kSlab, larger ones get a slab of their own without slack, and each goes to
// the slab that it fills best.  expect() sizes the first slab of a small arena (a 12^3 context holds 10 MB with
// everything, 96 MB while every arena began with a whole slab); beyond it a slab is a quarter of what the
// arena holds.  recycle() starts over in the slabs that are there, or gives them back where they hold more
// than kKeep, so that a large hierarchy does not outlive its solve; release() and the end free them.
class DevArena {
 public:
  static constexpr size_t kOwnSlab = (size_t)8 << 20, kSlab = (size_t)32 << 20, kKeep = (size_t)1 << 30;
  ~DevArena() { release(); }
  void expect(size_t bytes) { first_ = std::min(kSlab, round_up(bytes, (size_t)1 << 20)); }
  template <class T>
  T* alloc(size_t n) {
    const size_t want = round_up(std::max<size_t>(n, 1) * sizeof(T), 256);
    Slab* best = nullptr;
    for (Slab& s : slabs_)
      if (s.size - s.used >= want && (!best || s.size - s.used < best->size - best->used)) best = &s;
    if (!best) {
      const size_t share = std::min(kSlab, std::max(bytes_ == 0 ? first_ : (size_t)1 << 20, bytes_ / 4));
      Slab s;
      s.size = want >= kOwnSlab ? want : std::max(want, share);
      if (cudaMalloc(&s.ptr, s.size) != cudaSuccess) {  // no room for the spare part: the request alone
        cudaGetLastError();
        s.size = want;
        if (cudaMalloc(&s.ptr, s.size) != cudaSuccess) {
          cudaGetLastError();
          throw NoDeviceMemory(want);
        }
      }
      slabs_.push_back(s);
      bytes_ += s.size;
      best = &slabs_.back();
    }
    char* p = static_cast<char*>(best->ptr) + best->used;
    best->used += want;
    return reinterpret_cast<T*>(p);
  }
  template <class T>
  T* upload(const std::vector<T>& h) {
    T* d = alloc<T>(h.size());
    upload_now(d, h.data(), h.size() * sizeof(T));
    return d;
  }
  void recycle() {
    if (bytes_ > kKeep) return release();
    for (Slab& s : slabs_) s.used = 0;
  }
  void release() {
    for (Slab& s : slabs_) cudaFree(s.ptr);
    slabs_.clear();
    bytes_ = 0;
  }
  size_t bytes() const { return bytes_; }

 private:
  struct Slab {
    void* ptr = nullptr;
    size_t size = 0, used = 0;
  };
  static size_t round_up(size_t n, size_t to) { return (n + to - 1) / to * to; }
  std::vector<Slab> slabs_;
  size_t first_ = (size_t)1 << 20, bytes_ = 0;
};

// Runs make(), which fills a group of buffers from the arena, unless it is ready.  When an allocation fails
// half way the arena is given back and the group stays not ready, so that the next use starts afresh.
template <class F>
void build_once(bool& ready, DevArena& arena, F&& make) {
  if (ready) return;
  try {
    make();
  } catch (...) {
    arena.release();
    throw;
  }
  ready = true;
}

}  // namespace anb
