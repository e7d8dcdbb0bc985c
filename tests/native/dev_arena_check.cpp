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

  // a context's requests, from a few bytes to a share of a large grid: little is held beyond them, and a second
  // set of them in another order and a per cent smaller takes no more memory
  for (size_t cells : {(size_t)2000, (size_t)50000, (size_t)1000000}) {
    anb::DevArena b;
    b.expect(1300 * cells);
    size_t asked = 0, calls = g_blocks.size();
    const int per[] = {192, 4, 64, 24, 8, 8, 96, 1, 24, 53, 24, 8, 48, 512, 24, 24, 8, 8, 24, 24, 96, 24};
    for (int p : per) asked += p * cells, b.alloc<char>(p * cells);
    if (b.bytes() > asked * 1.1 + (3u << 20)) return fail("an arena holds far more than was asked for");
    if (g_blocks.size() - calls > 2 + (cells > 20000 ? 22 : 0)) return fail("a small arena took many allocations");
    const size_t held = g_held;
    b.recycle();
    for (int p : {512, 96, 96, 192, 64, 53, 48, 24, 24, 24, 24, 24, 24, 24, 8, 8, 8, 8, 4, 1})
      b.alloc<char>(p * cells * 99 / 100);
    if (b.bytes() <= anb::DevArena::kKeep && g_held > held) return fail("a recycled arena grew");
    b.release();
  }
  a.alloc<char>(anb::DevArena::kKeep / 2 + 1);
  a.alloc<char>(anb::DevArena::kKeep / 2 + 1);
  a.recycle();
  if (g_held) return fail("a large arena outlived its use");
  std::printf("ok\n");
  return 0;
}
