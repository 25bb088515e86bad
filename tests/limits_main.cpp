// Prints the limits of mg_limits.h for the sizes given on the command line.
#include <cstdio>
#include <cstdlib>
#include <cstring>

#include "mg_limits.h"

int main(int argc, char** argv) {
  auto arg = [&](int i) { return std::strtoull(i < argc ? argv[i] : "0", nullptr, 0); };
  const char* what = argc > 1 ? argv[1] : "";
  if (!std::strcmp(what, "lane_start")) {
    std::printf("%d\n", int(mg::lane_start(arg(2), arg(3), arg(4))));
    return 0;
  }
  if (!std::strcmp(what, "look_back")) {  // epoch, state, a, b: the word of a + b, taken apart
    const unsigned long long w =
        mg::lb_word(uint32_t(arg(2)), arg(3), mg::lb_sum(arg(4), arg(5)));
    std::printf("%u %llu %llu %llu %u\n", mg::lb_epoch(w), mg::lb_state(w), mg::lb_value(w),
                mg::LB_MAX, mg::LB_EPOCHS);
    return 0;
  }
  if (!std::strcmp(what, "emit_room")) {  // known, cap_rows, entries, limit, held, bytes of a row
    const unsigned long long row = arg(7);
    std::printf("%llu\n", (unsigned long long)mg::emit_room(
                              arg(2) != 0, arg(3), arg(4), arg(5), arg(6),
                              [&](uint64_t rows) { return rows * row; }));
    return 0;
  }
  if (!std::strcmp(what, "tables")) {  // used, cap, budget, rows of level 0, 1, ...
    uint64_t rows[16] = {};
    for (int l = 0; l < 16; ++l) rows[l] = arg(5 + l);
    const uint32_t mask = mg::tables_to_free(rows, 16, int(arg(2)), arg(3), arg(4),
                                             [](int l) { return uint64_t(l) * 4 + 21; });
    for (int l = 0; l < 16; ++l)
      if (mask >> l & 1u) std::printf("%d\n", l);
    return 0;
  }
  return 2;
}
