// Whether a caller's device array can be read by the index build's kernels where it is.
#pragma once

#include <cstddef>
#include <cstdint>

namespace fomo {

// `bytes` of floats at p, in an allocation of `size` bytes at `base`: aligned for 32-bit loads and whole in it.  A copy takes
// any address, and refuses one that runs past its allocation; a kernel does neither.
inline bool array_in_place(uintptr_t p, size_t bytes, uintptr_t base, size_t size) {
  return p % sizeof(float) == 0 && p >= base && p - base <= size && bytes <= size - (p - base);
}

}  // namespace fomo
