// march_split.h -- how many chunks along axis 0 a marching launch is cut into.
// Plain C++ (the rule is tested without a GPU).
//
// A CTA of a marching kernel takes planes + 2R steps for a chunk of `planes`
// planes.  The chip runs whole CTAs, `resident` per SM at a time, so a launch
// of 300 CTAs on 296 slots is two rounds, not 1.01.  Fitted to 34000 timed launches
// (complex128, float64 and float32, radius 1 to 3, grids of 24 to 144 points a
// side, 1 to 64 bands, every split; 5 to 10% rms): the steps cost the same
// throughout, and a last round that puts k of the `resident` CTAs on an SM costs
// 1/2 + k / (2 resident) of a full one, half of it being latency.  Priced by a
// fraction of a round instead, 30 bands of 66^3 took 144 steps where 112 do.
#pragma once

#include <algorithm>
#include <cstdint>

namespace gfd {

struct MarchSplit {
  int chunks;
  double steps;  // plane steps of the launch, rounds of CTAs times a CTA's steps
};

inline double march_rounds(int64_t ctas, int resident, int sms) {
  const int64_t slots = int64_t(resident) * sms, whole = ctas / slots, rest = ctas % slots;
  if (rest == 0) return double(whole);
  return double(whole) + 0.5 + 0.5 * double((rest + sms - 1) / sms) / resident;
}

// tiles: CTAs per chunk.  The chunk count with the fewest steps, the smaller of
// equals; chunks of at least 2R and 4 planes, and no more than 12 rounds of them
// (past that the 2R extra planes of each chunk outweigh an even tail).
inline MarchSplit march_split(int n0, int R, int64_t tiles, int resident, int sms) {
  const int64_t enough = 12LL * resident * sms / std::max<int64_t>(tiles, 1) + 1;
  const int most = int(std::min<int64_t>(std::max(1, n0 / std::max(4, 2 * R)), enough));
  MarchSplit best = {1, 0.0};
  for (int c = 1; c <= most; c++) {
    const int planes = (n0 + c - 1) / c;
    const int chunks = (n0 + planes - 1) / planes;
    const double steps = march_rounds(tiles * chunks, resident, sms) * (planes + 2 * R);
    if (c == 1 || steps < best.steps) best = {chunks, steps};
  }
  return best;
}

// The chunk count of a launch.  target > 0: that many CTAs per SM, of a launch
// plan or set for the process, whatever the rounds; else by march_split.
inline int march_chunks(int n0, int R, int64_t tiles, int resident, int sms, int target) {
  if (target <= 0) return march_split(n0, R, tiles, resident, sms).chunks;
  const int64_t want = (int64_t(target) * sms + tiles - 1) / tiles;
  const int most = std::max(1, n0 / std::max(4, 2 * R));
  return int(std::min<int64_t>(most, std::max<int64_t>(1, want)));
}

}  // namespace gfd
