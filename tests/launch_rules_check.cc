// Prints the planner's size rules (wmh_internal.h) for the arguments
// "row min_row evals", "filter s_pad samples nnz rows", "batch s_pad nnz rows", "keep s_pad spl
// tiny mean_row", "split total warps waves mean_row min_items" or "both s_pad rows".
#include <cstdio>
#include <cstdlib>
#include <cstring>

#include "wmh_internal.h"

int main(int argc, char **argv) {
  auto arg = [&](int i) { return i < argc ? strtoull(argv[i], nullptr, 10) : 0ull; };
  const uint32_t s_pad = static_cast<uint32_t>(arg(2));
  if (!strcmp(argv[1], "filter")) {
    printf("%d", mhb::filter_pays(s_pad, static_cast<uint32_t>(arg(3)), arg(4), arg(5)));
  } else if (!strcmp(argv[1], "batch")) {
    const mhb::FilterRule r = mhb::filter_rule(s_pad);
    printf("%d", arg(3) >= r.min_row * arg(4) && arg(3) >= r.min_batch / s_pad);
  } else if (!strcmp(argv[1], "keep")) {
    printf("%d", arg(5) < mhb::keep_rows(s_pad, static_cast<uint32_t>(arg(3)), arg(4) != 0));
  } else if (!strcmp(argv[1], "split")) {
    const mhb::FilterSplit p = mhb::filter_split(arg(2), arg(3), arg(4), arg(5), static_cast<uint32_t>(arg(6)));
    printf("%u %u", p.chunk, p.snap);
  } else if (!strcmp(argv[1], "row")) {
    printf("%llu", static_cast<unsigned long long>(mhb::filter_row(arg(2), arg(3))));
  } else if (!strcmp(argv[1], "both")) {
    printf("%d", arg(3) >= mhb::filter_batch_rows(s_pad));
  } else {
    return 2;
  }
  return 0;
}
