// device_buffers.h -- growth of a device buffer, free of CUDA: the allocator is a parameter.
#pragma once
#include <cstddef>

namespace ladds {

// p holds room for `need` elements afterwards, its contents are not kept.  The new
// buffer is taken before the old one is given back: where there is no memory for
// it, p and cap stay as they were -- a kernel launched later still finds the
// buffer it found before -- and the result is false.
// take(bytes): memory or null; give(p): returns it.
template <typename T, typename Take, typename Give>
bool growBuffer(T *&p, size_t &cap, size_t need, Take take, Give give) {
  if (p && need <= cap) return true;
  T *fresh = static_cast<T *>(take(need * sizeof(T)));
  if (!fresh) return false;
  if (p) give(p);
  p = fresh;
  cap = need;
  return true;
}

}  // namespace ladds
