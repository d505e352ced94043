// Prints, for offsets 0 to 15 of an array and elements of 4 and 8 bytes,
// whether the device may work on it in place.
#include <cstdio>

#include "host_access.h"

int main() {
  alignas(16) static char buf[64];
  for (size_t element : {4, 8})
    for (int off = 0; off < 16; ++off) {
      const void *a = buf + off, *b = buf + 16;
      std::printf("%zu %d %d%d%d%d%d\n", element, off, lbmpsm::in_place(true, element, {a}),
                  lbmpsm::in_place(true, element, {b, a}), lbmpsm::in_place(true, element, {a, nullptr, b}),
                  lbmpsm::in_place(true, element, {b, nullptr}), lbmpsm::in_place(false, element, {a}));
    }
}
