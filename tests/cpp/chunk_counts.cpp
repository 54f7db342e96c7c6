// counts_fit: where it holds, a count that grows by up to 32 (the warps of a
// block) every step stays in 31 bits over the whole run, and only runs that could
// leave them are turned down.
#include <cstdio>

#include "../../grn-gpu-performance_b200/csrc/grn_sim.h"

int main() {
  long wrong = 0;
  const int64_t limit = 0x7fffffff;
  for (int64_t n : {(int64_t)0, (int64_t)1, (int64_t)5000, (int64_t)1 << 25, limit / 32 - 1,
                    limit / 32, limit / 32 + 1, (int64_t)1 << 27, (int64_t)1 << 30, limit})
    if (grn::counts_fit((int)n) != (32 * n <= limit)) ++wrong;
  std::printf("wrong %ld\n", wrong);
  return wrong != 0;
}
