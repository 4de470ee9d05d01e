// The autotuner's candidates (tune_candidates.h): no two alike, the untuned configuration among them and first, radii
// varied alone, caps below the CTAs that fit.
#include <cstdio>

#include "tune_candidates.h"

int main() {
  int bad = 0;
  for (int ctas : {5, 7}) {
    const auto c = fomo::tune_candidates(ctas);
    auto is = [&](size_t i, int w, int h, int cap, float r) {
      return c[i].tile_w == w && c[i].tile_h == h && c[i].cap == cap && c[i].radius == r;
    };
    bad += !is(0, 8, 4, 0, 0.0f);
    for (size_t i = 0; i < c.size(); ++i) {
      for (size_t j = 0; j < i; ++j) bad += is(i, c[j].tile_w, c[j].tile_h, c[j].cap, c[j].radius);
      bad += c[i].cap != 0 && (c[i].cap < 1 || c[i].cap >= ctas);
      bad += c[i].radius != 0.0f && !is(i, 8, 4, 0, c[i].radius);
      bad += c[i].radius < 0.0f || c[i].tile_w * c[i].tile_h < 32;
    }
  }
  std::printf("%d\n", bad);
  return bad;
}
