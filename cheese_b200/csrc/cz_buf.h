// Work buffers that live as long as their context and grow on demand (host).
#pragma once
#include <algorithm>
#include <cstddef>

namespace cz {

// A buffer of Memory: Memory::get(bytes) returns a new block or throws, Memory::put(p) gives one back or throws,
// Memory::drop(p) gives one back and never throws. Contents are lost when it grows. Nothing is held from the old block's
// return until the new one is there, so after a failed call the buffer is empty and the next one allocates.
template <class Memory> struct GrowBuf {
  void *p = nullptr;
  size_t cap = 0;
  void ensure(size_t b) {
    if (b <= cap) return;
    const size_t c = (std::max(b, cap + cap / 2) + 255) & ~(size_t)255;
    void *old = p;
    p = nullptr;
    cap = 0;
    if (old) Memory::put(old);
    p = Memory::get(c);
    cap = c;
  }
  template <typename T> T *as() const { return (T *)p; }
  void release() {
    if (p) Memory::drop(p);
    p = nullptr;
    cap = 0;
  }
};

// releases what a call keeps for the next one unless the call came to its end: a failed call holds nothing
template <class Kept> struct ReleaseUnlessDone {
  Kept &kept;
  bool done = false;
  ~ReleaseUnlessDone() { if (!done) kept.release(); }
};

}  // namespace cz
