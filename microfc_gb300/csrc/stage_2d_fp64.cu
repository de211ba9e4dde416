// Instantiations of the fused stage kernel for 2-D cases, FP64 arithmetic.
// The first entry per configuration is the default until the autotuner runs:
// tiles sized for the grid (mfc_flex.cuh).
#include "mfc_launch.h"

namespace mfc {

void register_stage_2d_fp64(std::vector<StageEntry>& r) {
  r.push_back(flex_entry<2, 2, 5, 640>());
  // 32x16, interior tiles staged by one TMA bulk tensor copy: 1 % faster than
  // the sized tiles on the largest grids (15585 against 15761 us a step at
  // 2048x1024), 1 % slower at 1024x512
  r.push_back(stage_entry<2, 2, 5, double, 32, 16, 640, true>());
  r.push_back(flex_entry<2, 1, 5, 640>());
  r.push_back(flex_entry<2, 2, 3, 512>());
  r.push_back(flex_entry<2, 2, 1, 512>());
  r.push_back(flex_entry<2, 1, 3, 512>());
  r.push_back(flex_entry<2, 1, 1, 512>());
}

}  // namespace mfc
