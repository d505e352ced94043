// host_access.h -- when the device works on a caller's host arrays in place
// (coherent host memory) and when they are staged.  Host code only.
#pragma once

#include <cstddef>
#include <cstdint>
#include <initializer_list>

namespace lbmpsm {

// In place only where every array is aligned to its elements: a copy takes any
// address, a kernel's loads and stores fault on a misaligned one.  (NULL: not
// asked for.)
inline bool in_place(bool host_direct, size_t element, std::initializer_list<const void*> arrays) {
  for (const void* a : arrays)
    if (reinterpret_cast<uintptr_t>(a) % element != 0) return false;
  return host_direct;
}

}  // namespace lbmpsm
