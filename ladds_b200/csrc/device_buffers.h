// device_buffers.h -- growth and layout rules of device buffers, free of CUDA: the allocator is a parameter.
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

// whether a two-dimensional copy takes rows this many bytes apart: the driver
// refuses a pitch above 2^31 - 1 (cudaDeviceProp::memPitch), which arrays of
// 2^28 - 1 doubles in 256-byte steps exceed
constexpr bool copyPitchFits(size_t bytes) { return bytes <= ((size_t)1 << 31) - 1; }

}  // namespace ladds
