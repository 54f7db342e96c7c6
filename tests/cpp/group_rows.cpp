// Rows of float4 groups as the simulation kernel finds them
// (group_row, with set_geometry's constants) against integer division, for
// every group of the grids "W H" on the command line: the strips of two rows
// and the rows of the initial state with their border rows.  Prints the
// groups that differ.
#include <cstdio>
#include <cstdlib>

#include "../../grn-gpu-performance_b200/csrc/grn_sim.h"

int main(int argc, char **argv) {
  long wrong = 0;
  for (int k = 1; k + 1 < argc; k += 2) {
    const int W = std::atoi(argv[k]), H = std::atoi(argv[k + 1]);
    grn::SimArgs a{};
    grn::set_geometry(&a, W, H, 1, 0);
    for (long i = 0; i < (long)(H + 3) * a.Wg; ++i) {
      const int row = grn::group_row((int)i, a.Wg, a.inv_wg, a.wg_shift);
      if (row == i / a.Wg) continue;
      if (wrong++ < 5) std::printf("%d x %d: group %ld in row %d\n", W, H, i, row);
    }
  }
  std::printf("wrong %ld\n", wrong);
  return wrong != 0;
}
