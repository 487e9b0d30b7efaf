// The host side of nsp_b200/csrc/runrules.h, for tests/test_run_rules_cpu.py.
#include "runrules.h"

using namespace nspb;

extern "C" {

int max_a(void) { return kRunMaxA; }
int max_ip(void) { return kRunMaxIp; }

// Products of a row as the kernels add them: 32 lengths at a time in 32 bits, and
// no further once there are too many.
int row_products(const int *len, int na) {
  int total = 0;
  for (int c = 0; c < na; c += 32) {
    unsigned sum = 0;
    for (int t = c; t < na && t < c + 32; ++t) sum += (unsigned)run_len(len[t]);
    total += (int)sum;
    if (total > kRunMaxIp) return kRunMaxIp + 1;
  }
  return total;
}
}
