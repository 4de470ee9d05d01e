// Which device arrays the index build reads where they are (array_in_place.h).
#include <cstdio>

#include "array_in_place.h"

int main() {
  const uintptr_t b = 0x7f0000000000;
  const struct {
    uintptr_t p;
    size_t bytes;
    bool in_place;
  } cases[] = {
      {b, 4096, true},        {b + 4, 4092, true},  {b + 4092, 4, true},     {b, 4, true},
      {b + 1, 4, false},      {b + 2, 64, false},   {b + 3, 4092, false},    // misaligned
      {b, 4100, false},       {b + 8, 4092, false}, {b + 4096, 4, false},    // past the end
      {b + 8192, 4, false},   {b - 4, 8, false},    {b, ~size_t(0) - 3, false},
  };
  int bad = 0;
  for (const auto& c : cases)
    if (fomo::array_in_place(c.p, c.bytes, b, 4096) != c.in_place) {
      std::printf("offset %lld, %zu bytes: %d\n", (long long)(c.p - b), c.bytes, !c.in_place);
      ++bad;
    }
  return bad;
}
