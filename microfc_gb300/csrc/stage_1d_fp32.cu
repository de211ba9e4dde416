// Instantiations of the fused stage kernel for 1-D cases, split precision.
#include "mfc_launch.h"

namespace mfc {

void register_stage_1d_fp32(std::vector<StageEntry>& r) {
  r.push_back(stage_entry<1, 1, 1, float, 128, 1, 128>());
  r.push_back(stage_entry<1, 1, 3, float, 128, 1, 128>());
  r.push_back(stage_entry<1, 2, 1, float, 128, 1, 128>());
  r.push_back(stage_entry<1, 2, 3, float, 128, 1, 128>());
  // 62 cells: 64 positions, a run of two of one of three pairs for each of 96 threads
  r.push_back(pair_entry<1, 1, 62, 1, 96, 10, 2, 1>());
  r.push_back(pair_entry<1, 2, 62, 1, 96, 10, 2, 1>());
}

}  // namespace mfc
