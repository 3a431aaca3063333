// Shape of the assembly launch: vertices per CTA (128, or 64 for the small shape's
// 32) and lanes per vertex.
#pragma once

#include <cstdint>

namespace bartels {

struct HessShape {
  int chunk, lanes;
};

// The lanes follow from the size, so that the values do not depend on the tuning;
// the shape is the plan's tuning where it has one (0: none).
//
// Four lanes while a vertex's pair of lanes would leave most SMs short of work
// (15.6k vertices: 31 us, two lanes 38). The cheap laws' one-lane form runs in
// one wave of three 128-vertex chunks per SM, so its time hardly grows up to
// there; the two-lane form's second wave starts at ~190 vertices per SM on a
// mesh numbered without locality. Shuffled balls, one lane / two: 27.6k
// vertices 66 / 60 us, 30.1k 67 / 72, 37.5k 67 / 78, 56.2k 94 / 112, 63.4k (a
// second wave) 153 / 128. On a mesh numbered with locality the lines cross later
// (boxes: 35.9k 52 / 43, 50.7k 64 / 69, 59.3k 96 / 72): below ~45k vertices a box
// gives up to 20% for the shuffled meshes' sake.
inline HessShape hess_shape(int64_t vertices, int64_t chunks128, int64_t sms, bool cheap, int tuned) {
  const bool one = cheap && vertices > 190 * sms && chunks128 <= 3 * sms;
  return {tuned ? tuned : one ? 128 : 64, one ? 1 : vertices <= 128 * sms ? 4 : 2};
}

}  // namespace bartels
