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

// Device allocations owned by a context, cut from slabs and given back together.  recycle() starts
// over in the slabs that are there (a hierarchy rebuilt for every solve made ~60 cudaMalloc / cudaFree
// pairs a time, 8 ms on the freeing side alone); release() and the end of the context free them.  A slab
// is at least 32 MB or a quarter of what the arena holds, at most 1 GB beyond a larger request.
class DevArena {
 public:
  ~DevArena() { release(); }
  template <class T>
  T* alloc(size_t n) {
    const size_t want = (std::max<size_t>(n, 1) * sizeof(T) + 255) & ~(size_t)255;
    for (; cur_ < slabs_.size(); ++cur_, used_ = 0)
      if (used_ + want <= slabs_[cur_].size) break;
    if (cur_ == slabs_.size()) {
      Slab s;
      s.size = std::max(want, std::min(std::max((size_t)32 << 20, bytes_ / 4), (size_t)1 << 30));
      if (cudaMalloc(&s.ptr, s.size) != cudaSuccess) {  // no room for the spare part: the request alone
        cudaGetLastError();
        s.size = want;
        CK(cudaMalloc(&s.ptr, s.size));
      }
      slabs_.push_back(s);
      bytes_ += s.size;
      used_ = 0;
    }
    char* p = static_cast<char*>(slabs_[cur_].ptr) + used_;
    used_ += want;
    return reinterpret_cast<T*>(p);
  }
  template <class T>
  T* upload(const std::vector<T>& h) {
    T* d = alloc<T>(h.size());
    upload_now(d, h.data(), h.size() * sizeof(T));
    return d;
  }
  void recycle() { cur_ = used_ = 0; }
  void release() {
    for (Slab& s : slabs_) cudaFree(s.ptr);
    slabs_.clear();
    cur_ = used_ = bytes_ = 0;
  }
  size_t bytes() const { return bytes_; }

 private:
  struct Slab {
    void* ptr = nullptr;
    size_t size = 0;
  };
  std::vector<Slab> slabs_;
  size_t cur_ = 0, used_ = 0, bytes_ = 0;
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
