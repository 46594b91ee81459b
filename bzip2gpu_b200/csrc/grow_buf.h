// Scratch that only grows (contents are not kept), with the allocator as a
// parameter: Mem::alloc gives nullptr where memory is short.
#pragma once

#include <stddef.h>

#include <algorithm>

namespace bz2g {

template <class Mem>
struct GrowBuf {
  void *p = nullptr;
  size_t cap = 0;
  template <typename T>
  T *get() const {
    return static_cast<T *>(p);
  }
  void release() {
    if (p) Mem::free(p);
    p = nullptr;
    cap = 0;
  }
  // false: memory is short; the buffer is then empty
  bool try_reserve(size_t bytes) {
    bytes = std::max<size_t>(bytes, 16);
    if (bytes <= cap) return true;
    release();
    p = Mem::alloc(bytes);
    if (p) cap = bytes;
    return p != nullptr;
  }
};

// Reserves b, giving up `spare` (scratch that its user can do without) where
// memory is short.
template <class Mem>
bool reserve_or_free(GrowBuf<Mem> &b, size_t bytes, GrowBuf<Mem> &spare) {
  if (b.try_reserve(bytes)) return true;
  if (&b == &spare || !spare.cap) return false;
  spare.release();
  return b.try_reserve(bytes);
}

}  // namespace bz2g
