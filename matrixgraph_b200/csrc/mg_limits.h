// Limits of an enumeration call as plain functions of sizes, so that they can be
// checked at sizes that no test could put on a device.
#pragma once

#include <cstdint>

namespace mg {

// What a batch lane does with a query of t0 level-0 candidates.  Its expand
// launch covers at most seg_cap elements; at the later levels k_work_scan flags a
// larger total, but level 0 has no such launch, so the host decides.
enum class LaneStart {
  kRun,      // levels are queued on the lane
  kUnknown,  // past the per-query budget (0: none) before anything has run
  kChunked,  // too large for a lane: counted on the chunked path
};
inline LaneStart lane_start(uint64_t t0, uint64_t budget, uint64_t seg_cap) {
  if (budget && t0 > budget) return LaneStart::kUnknown;
  return t0 > seg_cap ? LaneStart::kChunked : LaneStart::kRun;
}

}  // namespace mg
