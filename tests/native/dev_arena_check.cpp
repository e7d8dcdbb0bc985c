// CPU check of csrc/dev_arena.hpp on a stand-in for the CUDA runtime whose cudaMemcpy returns with the copy
// still queued, as the real one may for pageable memory; only cudaStreamSynchronize(cudaStreamLegacy) or a
// later copy lands it.  Prints "ok" or what failed.
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <numeric>

#include "../../anabasis_b200/csrc/dev_arena.hpp"

static struct {
  void* dst;
  std::vector<char> data;
} g_queued;
static size_t g_held = 0, g_limit = ~(size_t)0;
static std::vector<std::pair<void*, size_t>> g_blocks;

static void land() {
  if (!g_queued.data.empty()) std::memcpy(g_queued.dst, g_queued.data.data(), g_queued.data.size());
  g_queued.data.clear();
}

extern "C" {
cudaError_t CUDARTAPI cudaMalloc(void** p, size_t n) {
  if (g_held + n > g_limit || !(*p = std::aligned_alloc(256, (n + 255) & ~(size_t)255))) return cudaErrorMemoryAllocation;
  std::memset(*p, 0xee, n);
  g_held += n;
  g_blocks.push_back({*p, n});
  return cudaSuccess;
}
cudaError_t CUDARTAPI cudaFree(void* p) {
  for (auto& b : g_blocks)
    if (b.first == p) {
      g_held -= b.second;
      b = g_blocks.back();
      g_blocks.pop_back();
      break;
    }
  std::free(p);
  return cudaSuccess;
}
cudaError_t CUDARTAPI cudaMemcpy(void* dst, const void* src, size_t n, cudaMemcpyKind) {
  land();
  g_queued.dst = dst;
  g_queued.data.assign((const char*)src, (const char*)src + n);
  return cudaSuccess;
}
cudaError_t CUDARTAPI cudaStreamSynchronize(cudaStream_t s) {
  if (s == cudaStreamLegacy) land();
  return cudaSuccess;
}
cudaError_t CUDARTAPI cudaGetLastError(void) { return cudaSuccess; }
const char* CUDARTAPI cudaGetErrorString(cudaError_t) { return "out of memory"; }
}

static int fail(const char* what) {
  std::printf("%s\n", what);
  return 1;
}

int main() {
  anb::DevArena a;
  std::vector<int> h(100003);
  std::iota(h.begin(), h.end(), 7);
  const int* d = a.upload(h);
  if (std::memcmp(d, h.data(), h.size() * sizeof(int))) return fail("an upload returned before its data had landed");
  if (a.upload(std::vector<int>()) == nullptr) return fail("empty upload");
  const char* lo = (const char*)a.alloc<char>(1);
  const char* hi = (const char*)a.alloc<double>(3);
  if (((size_t)lo | (size_t)hi) & 255) return fail("alignment");
  if (hi < lo + 256) return fail("overlap");
  if (std::memcmp(d, h.data(), h.size() * sizeof(int))) return fail("an earlier upload was overwritten");
  a.release();
  if (g_held) return fail("release left memory behind");

  // a group of buffers whose second allocation fails: not ready, nothing held, made anew later
  bool ready = false;
  const void *first = nullptr, *second = nullptr;
  auto make = [&] {
    first = a.alloc<char>((size_t)64 << 20);
    second = a.alloc<char>((size_t)96 << 20);
  };
  g_limit = (size_t)128 << 20;
  bool threw = false;
  try {
    anb::build_once(ready, a, make);
  } catch (const anb::AnbError& e) {
    threw = e.code == ANB_ERR_CUDA;
  }
  if (!threw || ready || second || g_held) return fail("a failed group was kept");
  g_limit = ~(size_t)0;
  first = nullptr;
  anb::build_once(ready, a, make);
  if (!ready || !first || !second) return fail("a failed group was not made anew");
  const void* was = first;
  anb::build_once(ready, a, make);
  if (first != was) return fail("a ready group was made twice");
  a.release();
  std::printf("ok\n");
  return 0;
}
