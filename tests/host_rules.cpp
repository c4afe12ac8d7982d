// Prints what the library's host rules (csrc/xpcs_internal.h) give, one value
// per line, for tests/test_host_rules.py.  No device is touched.
//   host_rules hist N ...      words of the radix sorts' histogram for N items
#include <cstdio>
#include <cstdlib>
#include <cstring>

#include "xpcs_internal.h"

int main(int argc, char **argv) {
  if (argc > 1 && !std::strcmp(argv[1], "hist"))
    for (int k = 2; k < argc; k++)
      std::printf("%zu\n", xg::radix_hist_words(std::atoll(argv[k])));
  return 0;
}
