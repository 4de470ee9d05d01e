// The march configurations that the autotuner measures.
#pragma once

#include <vector>

namespace fomo {

// cap: CTAs per SM of the search, 0 for as many as fit; radius: gather radius in local point spacings, 0 for the cloud's
// own default.
struct TuneCandidate {
  int tile_w, tile_h, cap;
  float radius;
};

// `ctas`: CTAs per SM of the search that most of the batch's views take.  The untuned configuration first, then the ray tiles
// and caps that bind that search at the default radius, and radii on either side of the defaults (0.87 and 1.1) at the
// default tile.  A tile of one row holds no 2 x 2 blocks: its views are searched one ray per warp.
inline std::vector<TuneCandidate> tune_candidates(int ctas) {
  return {{8, 4, 0, 0.0f},        {16, 2, 0, 0.0f},       {4, 8, 0, 0.0f}, {32, 1, 0, 0.0f}, {8, 8, 0, 0.0f},
          {8, 4, ctas - 1, 0.0f}, {8, 4, ctas - 2, 0.0f}, {8, 4, 0, 0.8f}, {8, 4, 0, 1.0f},  {8, 4, 0, 1.2f}};
}

}  // namespace fomo
