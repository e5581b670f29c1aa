// Places in a block of page-locked memory that the host fills, one call behind another, and kernels read later.  Plain C++: no
// CUDA, so that the arithmetic can be checked on its own.
#pragma once

#include <cstddef>

namespace relux {

struct HostRing {
  size_t size = 0, used = 0;
  static size_t padded(size_t bytes) { return (bytes + 255) & ~(size_t)255; }
  // Places for the n pieces of one call, all at once: at[i] is the offset of bytes[i].  Where they do not fit behind the pieces of the
  // calls before, wait() is called first and the places start again: it returns once the kernels of every call before this one are
  // complete (false: it failed, and nothing is taken).  Taken piece by piece, the wait could fall between two pieces of a call, when
  // the call's own kernel was not queued yet, and the first piece was handed out again a turn later without another wait.
  template <class Wait>
  bool take(const size_t* bytes, int n, size_t* at, Wait wait) {
    size_t need = 0;
    for (int i = 0; i < n; i++) need += padded(bytes[i]);
    if (need > size) return false;
    if (need > size - used) {
      if (!wait()) return false;
      used = 0;
    }
    for (int i = 0; i < n; i++) {
      at[i] = used;
      used += padded(bytes[i]);
    }
    return true;
  }
  // Everything queued so far is complete.
  void restart() { used = 0; }
};

}  // namespace relux
