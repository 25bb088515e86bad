// Limits of an enumeration call as plain functions of sizes, so that they can be
// checked at sizes that no test could put on a device.
#pragma once

#include <cstdint>

#ifdef __CUDACC__
#define MG_HD __host__ __device__ __forceinline__
#else
#define MG_HD inline
#endif

namespace mg {

// Look-back words of the single-pass work/scan: [epoch:8 | state:2 | value:54].
// A level's element total can pass 2^42 in ordinary use (a position that is not
// joined to the one before it), so the value has what the epoch does not need;
// the words are cleared when the epochs run out.  Sums stay at LB_MAX once they
// reach it, which no walk could expand anyway (days at 10^11 elements/s).
constexpr int LB_VALUE_BITS = 54;
constexpr uint32_t LB_EPOCHS = (1u << (62 - LB_VALUE_BITS)) - 1;  // 1..LB_EPOCHS
constexpr unsigned long long LB_AGG = 1, LB_INC = 2;  // a tile's sum, sum up to it
constexpr unsigned long long LB_MAX = (1ull << LB_VALUE_BITS) - 1;

// a + b, at most LB_MAX (a and b themselves may be any sums below 2^63).
MG_HD unsigned long long lb_sum(unsigned long long a, unsigned long long b) {
  const unsigned long long s = a + b;
  return s < LB_MAX ? s : LB_MAX;
}
MG_HD unsigned long long lb_word(uint32_t epoch, unsigned long long state, unsigned long long v) {
  return (unsigned long long)(epoch) << (LB_VALUE_BITS + 2) | state << LB_VALUE_BITS | v;
}
MG_HD uint32_t lb_epoch(unsigned long long w) { return uint32_t(w >> (LB_VALUE_BITS + 2)); }
MG_HD unsigned long long lb_state(unsigned long long w) { return w >> LB_VALUE_BITS & 3ull; }
MG_HD unsigned long long lb_value(unsigned long long w) { return w & LB_MAX; }

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

// Level tables to give back (a bit per level) before a call that uses levels
// 1..used-1 with up to cap rows each may grow its own: none when what it will hold
// at most, with the tables that earlier calls left, is within the budget; else
// those of levels it does not use and those of more than cap rows.  rows[l]: rows
// that table l has now; row_bytes(l): bytes of a row.  cap rows of every used
// level are within the budget.
template <class RowBytes>
inline uint32_t tables_to_free(const uint64_t* rows, int levels, int used, uint64_t cap,
                               uint64_t budget, RowBytes row_bytes) {
  uint64_t most = 0;
  uint32_t mask = 0;
  for (int l = 1; l < levels; ++l) {
    most += (l < used && rows[l] < cap ? cap : rows[l]) * row_bytes(l);
    if (rows[l] && (l >= used || rows[l] > cap)) mask |= 1u << l;
  }
  return most > budget ? mask : 0;
}

// Rows that an emit call makes room for before it knows how many there are, or 0:
// count first.  The caller has memory for cap_rows rows (known), or takes any
// number.  bytes(rows): size of the buffer; limit: bytes it may take; held: bytes
// that an earlier call left with the graph.
//   known    A buffer of up to `limit` is tried at its full size, so that what
//            fits the caller is enumerated once; a larger one is counted first,
//            since an attempt at less than the caller's room would be a third
//            enumeration of just those results that are large.
//   unknown  Room as the level tables start: by the graph's entries (vertices and
//            adjacency), so that ten rows of a small graph do not take 130 MB, and
//            as much as the block that is there holds anyway.
constexpr uint64_t kEmitTryMin = 1ull << 16, kEmitTry = 1ull << 22;

template <class Bytes>
inline uint64_t emit_room(bool known, uint64_t cap_rows, uint64_t entries, uint64_t limit,
                          uint64_t held, Bytes bytes) {
  uint64_t room = kEmitTryMin;
  if (known) {
    if (cap_rows >= 1ull << 31) return 0;
    if (cap_rows > room) room = cap_rows;
  } else {
    while (room < kEmitTry && ((room < 4 * entries && bytes(2 * room) <= limit) ||
                               bytes(2 * room) <= held))
      room <<= 1;
  }
  return bytes(room) <= limit || bytes(room) <= held ? room : 0;
}

}  // namespace mg
