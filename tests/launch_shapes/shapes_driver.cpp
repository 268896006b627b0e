// Driver for tests/test_launch_shapes.py: the launch shapes of the autotuner's
// candidates (no GPU).
#include "../../xara_gb300/csrc/xg_internal.h"

extern "C" int grid_of(int n, int nblk, int kb, int rows, int most) {
  return xg::pcg_grid(n, nblk, kb, rows, most);
}
