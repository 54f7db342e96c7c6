// count_reached over whole runs of 2^31 - 1 steps, around every step where a
// count or its target passes a power of two: behind by one part, level, and
// ahead by up to two steps.
#include <cstdio>

#include "../../grn-gpu-performance_b200/csrc/grn_sim.h"

int main() {
  long wrong = 0, tried = 0;
  for (int64_t per_step = 1; per_step <= 32; ++per_step)
    for (int b = 0; b <= 36; ++b)
      for (int64_t d = -3; d <= 3; ++d) {
        const int64_t step = ((int64_t)1 << b) / per_step + d;
        if (step < 1 || step > 0x7fffffff) continue;
        const int64_t target = per_step * step;
        for (int64_t ahead = -2 * per_step; ahead <= 2 * per_step; ++ahead) {
          if (target + ahead < 0) continue;
          ++tried;
          if (grn::count_reached((uint32_t)(target + ahead), (uint32_t)target) != (ahead >= 0))
            ++wrong;
        }
      }
  std::printf("tried %ld wrong %ld\n", tried, wrong);
  return wrong != 0 || tried == 0;
}
