// Time estimate behind the launch shapes of the NO_REF_DEL sweeps (host side).
#pragma once

#include <algorithm>
#include <cmath>
#include <cstdint>

#include "dtwx_internal.h"

namespace dtwx {

// What a strip's row of a sweep kernel costs, in cycles of one SM sub-partition:
// of a warp that has it to itself, and of each of several warps that share it.
// The second is the rate of a full GPU (FP16 pairs 17.8 Tcell/s at 48 cells per
// lane, FP32 12.9 at 48, MIXED 13.9 at 64), the first comes from one-read batches.
struct RowCost {
  int S;
  double alone, shared;
};
constexpr RowCost kFp16RowCost = {48, 265, 217};  // (the estimate is of FP32 and MIXED shapes)
constexpr RowCost kRowCost[3][3] = {{},
                                    {{16, 150, 65}, {32, 230, 111}, {48, 290, 152}},
                                    {{32, 260, 115}, {48, 320, 148}, {64, 360, 184}}};

// Estimated time (in cycles) of a NO_REF_DEL sweep of `items` equal work items
// on `teams` CTAs of k warps: an item is `work` strips' worth of rows in
// `strips` strips.  The warps of a CTA sweep strips as a pipeline, each one
// 32-row window behind its left neighbour, and share the SM's schedulers; both
// limits are real at once near the middle, so they add in squares (within 10 %
// of 270 measured shapes of eight batches, FP32 and MIXED cells).
inline double sweep_estimate(const RowCost &c, int64_t items, double work, double strips, double rows, int k,
                             int64_t teams, int sms) {
  const double per_team = std::ceil((double)items / (double)teams) * work;
  const double alone = c.alone * (rows * std::max(1.0, per_team / k) + kWarp * (std::min(strips, (double)k) - 1.0));
  const double ctas_per_sm = (double)teams / sms;
  const double used = std::min(1.0, (double)items / (double)teams);
  const double shared = per_team * rows * c.shared / 4.0 * std::max(1.0, ctas_per_sm * used);
  return std::sqrt(alone * alone + shared * shared);
}

}  // namespace dtwx
