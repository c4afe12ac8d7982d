// Prints what the library's host rules (csrc/xpcs_internal.h) give, one value
// per line, for tests/test_host_rules.py.  No device is touched.
//   host_rules hist N ...      words of the radix sorts' histogram for N items
//   host_rules rows P E F      rows the caller holds, P pixels, E events, F frames:
//                              thread kernel's row capacity, and the longest row that
//                              a series takes by thread (0: every row to a warp)
//   host_rules tuned P E F T   the same longest row alone and in a batch, of a tuned
//                              series of capacity 48 that keeps (T = 1) the thread kernel
#include <cstdio>
#include <cstdlib>
#include <cstring>

#include "xpcs_internal.h"

int main(int argc, char **argv) {
  if (argc > 1 && !std::strcmp(argv[1], "hist"))
    for (int k = 2; k < argc; k++)
      std::printf("%zu\n", xg::radix_hist_words(std::atoll(argv[k])));
  if (argc == 5 && !std::strcmp(argv[1], "rows")) {
    xg::Series s;
    s.P = std::atoi(argv[2]);
    s.raw_events = std::atoll(argv[3]);
    s.F = std::atoi(argv[4]);
    xg::default_knobs(s, true);
    std::printf("%d\n%d\n", s.thread_cap, s.class_cap);
  }
  if (argc == 6 && !std::strcmp(argv[1], "tuned")) {
    xg::Series s;
    s.P = std::atoi(argv[2]);
    s.raw_events = std::atoll(argv[3]);
    s.F = std::atoi(argv[4]);
    s.thread_cap = 48;
    s.knobs_set = s.tuned = true;
    s.by_thread = std::atoi(argv[5]) != 0;
    for (bool alone : {true, false}) {
      xg::default_knobs(s, alone);
      std::printf("%d\n", s.class_cap);
    }
  }
  return 0;
}
