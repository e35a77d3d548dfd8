// Growth of a device buffer with an allocator that runs out of memory; the
// distance of arrays that one two-dimensional copy can take.
#include "device_buffers.h"

#include <cassert>
#include <cstdint>
#include <cstdio>
#include <cstdlib>

int main() {
  size_t held = 0, limit = 1000;
  auto take = [&](size_t bytes) -> void * {
    if (held + bytes > limit) return nullptr;
    held += bytes;
    auto *p = static_cast<size_t *>(std::malloc(sizeof(size_t) + bytes));
    *p = bytes;
    return p + 1;
  };
  auto give = [&](void *p) {
    size_t *q = static_cast<size_t *>(p) - 1;
    held -= *q;
    std::free(q);
  };
  uint32_t *p = nullptr;
  size_t cap = 0;
  assert(ladds::growBuffer(p, cap, 100, take, give) && p && cap == 100 && held == 400);
  uint32_t *const first = p;
  assert(ladds::growBuffer(p, cap, 60, take, give) && p == first && cap == 100);
  // no memory for the larger one: the buffer in hand stays, and stays usable
  assert(!ladds::growBuffer(p, cap, 151, take, give) && p == first && cap == 100 && held == 400);
  p[99] = 7;
  assert(ladds::growBuffer(p, cap, 100, take, give) && p == first && p[99] == 7);
  assert(ladds::growBuffer(p, cap, 150, take, give) && p != first && cap == 150 && held == 600);
  give(p);
  assert(held == 0);
  // arrays of the largest population (28-bit slots), each on a 256-byte boundary
  const size_t apart = ((((size_t)1 << 28) - 1) * sizeof(double) + 255) / 256 * 256;
  assert(!ladds::copyPitchFits(apart) && ladds::copyPitchFits(apart - 256) && ladds::copyPitchFits(8));
  std::puts("device_buffers: ok");
  return 0;
}
