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
  return 2;
}
