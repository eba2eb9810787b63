// devbuf.cu -- growable device buffers, alone or several in one allocation.
#include <cuda_runtime.h>

#include <algorithm>

#include "internal.h"

namespace bude {

static int allocate(std::shared_ptr<void> &block, size_t nbytes, const char *what) {
  void *p = nullptr;
  const cudaError_t e = cudaMalloc(&p, std::max<size_t>(nbytes, 256));
  if (e != cudaSuccess) {
    cudaGetLastError(); // a caller may do with less
    return cuda_error(e, what);
  }
  block = std::shared_ptr<void>(p, [](void *q) { cudaFree(q); });
  return BUDE_OK;
}

int DevBuf::reserve(size_t nbytes, const char *what) {
  if (nbytes <= cap) return BUDE_OK;
  release();
  const int rc = allocate(block, nbytes, what);
  if (rc) return rc;
  ptr = block.get();
  cap = nbytes;
  return BUDE_OK;
}

void DevBuf::release() {
  block.reset();
  ptr = nullptr;
  cap = 0;
}

// The old block goes before the new one comes, and as a whole: a block lives as long as any buffer in it, so
// one that stayed would hold the outgrown ones' memory too.  No buffer gets smaller where there is room:
// uploads that take turns in what is large do not allocate each time.
int reserve_together(std::initializer_list<DevWant> wants, const char *what) {
  auto room = [](size_t bytes) { return (bytes + 511) / 512 * 512; };
  bool enough = true;
  size_t least = 0, most = 0;
  for (const DevWant &w : wants) {
    enough = enough && w.bytes <= w.buf->cap;
    least += room(w.bytes);
    most += room(std::max(w.bytes, w.buf->cap));
  }
  if (enough) return BUDE_OK;
  std::vector<size_t> bytes;
  for (const DevWant &w : wants) {
    bytes.push_back(std::max(w.bytes, w.buf->cap));
    w.buf->release();
  }
  std::shared_ptr<void> block;
  int rc = allocate(block, most, what);
  if (rc && least < most) {
    bytes.clear();
    for (const DevWant &w : wants) bytes.push_back(w.bytes);
    rc = allocate(block, least, what);
  }
  if (rc) return rc;
  size_t at = 0, i = 0;
  for (const DevWant &w : wants) {
    const size_t n = bytes[i++];
    if (n == 0) continue;
    w.buf->block = block;
    w.buf->ptr = static_cast<unsigned char *>(block.get()) + at;
    w.buf->cap = n;
    at += room(n);
  }
  return BUDE_OK;
}

} // namespace bude
