// devbuf_check.cpp -- the device buffers of csrc/devbuf.cu over a counted heap in place of cudaMalloc.
#include <cstdio>
#include <cstdlib>
#include <map>

#include "internal.h"

static size_t g_limit = 1 << 30, g_held = 0, g_peak = 0, g_calls = 0;
static std::map<void *, size_t> g_blocks;

extern "C" cudaError_t cudaMalloc(void **p, size_t n) {
  ++g_calls;
  if (g_held + n > g_limit) return cudaErrorMemoryAllocation;
  *p = std::aligned_alloc(512, (n + 511) / 512 * 512);
  g_blocks[*p] = n;
  g_held += n;
  g_peak = g_held > g_peak ? g_held : g_peak;
  return cudaSuccess;
}

extern "C" cudaError_t cudaFree(void *p) {
  g_held -= g_blocks.at(p);
  g_blocks.erase(p);
  std::free(p);
  return cudaSuccess;
}

extern "C" cudaError_t cudaGetLastError() { return cudaSuccess; }

namespace bude {
int cuda_error(cudaError_t, const char *) { return BUDE_ERR_CUDA; }
} // namespace bude

using bude::DevBuf;

#define CHECK(x)                                            \
  if (!(x)) {                                               \
    std::printf("line %d: %s\n", __LINE__, #x);             \
    return 1;                                               \
  }

int main() {
  constexpr size_t kOnce = 4096, kMost = 1 << 20;
  {
    // A group of which one buffer never grows: what the others outgrow is given back.
    DevBuf poses, energies, rows;
    size_t last = 0;
    for (size_t n = 1000; n <= kMost; n = n * 3 / 2) {
      CHECK(!bude::reserve_together({{&poses, 24 * n}, {&energies, 4 * n}, {&rows, kOnce}}, "group"));
      CHECK(g_held <= 28 * n + kOnce + 3 * 512);
      CHECK(g_peak <= 28 * n + kOnce + 3 * 512);
      CHECK(poses.cap >= 24 * n && energies.cap >= 4 * n && rows.cap >= kOnce);
      unsigned char *p = poses.as<unsigned char>(), *e = energies.as<unsigned char>(), *r = rows.as<unsigned char>();
      CHECK(p + poses.cap <= e || e + energies.cap <= p);
      CHECK(e + energies.cap <= r || r + rows.cap <= e);
      CHECK(g_blocks.size() == 1);
      last = n;
    }
    // Fewer poses, and the same again: nothing is allocated.
    const size_t calls = g_calls;
    CHECK(!bude::reserve_together({{&poses, 24}, {&energies, 4}, {&rows, kOnce}}, "group"));
    CHECK(!bude::reserve_together({{&poses, 24 * last}, {&energies, 4 * last}, {&rows, kOnce}}, "group"));
    CHECK(g_calls == calls);
    // A buffer that grew alone joins the group again with what it has.
    CHECK(!energies.reserve(64 * last, "alone"));
    CHECK(!bude::reserve_together({{&poses, 25 * last}, {&energies, 4 * last}, {&rows, kOnce}}, "group"));
    CHECK(g_blocks.size() == 1 && energies.cap >= 64 * last);
    // Where there is no room for that, with what is asked for.
    g_limit = 50 * last;
    CHECK(!bude::reserve_together({{&poses, 30 * last}, {&energies, 4 * last}, {&rows, kOnce}}, "group"));
    CHECK(poses.cap == 30 * last && energies.cap == 4 * last && g_blocks.size() == 1);
    // One that cannot be had leaves no buffer that looks reserved.
    CHECK(bude::reserve_together({{&poses, 50 * last}, {&energies, 4 * last}, {&rows, kOnce}}, "group"));
    CHECK(!poses.ptr && !energies.ptr && !rows.ptr && poses.cap + energies.cap + rows.cap == 0 && g_held == 0);
    g_limit = 1 << 30;
    CHECK(!bude::reserve_together({{&poses, 24}, {&energies, 0}, {&rows, kOnce}}, "group"));
    CHECK(poses.ptr && !energies.ptr && rows.ptr);
  }
  CHECK(g_held == 0);
  std::puts("ok");
  return 0;
}
