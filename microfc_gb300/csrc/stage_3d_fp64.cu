// Instantiations of the 3-D directional sweeps, FP64 arithmetic.
#include "mfc_launch.h"

namespace mfc {

void register_stage_3d_fp64(std::vector<StageEntry>& r) {
  r.push_back(flex_sweep_entry<2, 5, 640>());
  // fixed tiles, TMA-staged: even with the sized ones where the grid is a
  // multiple of both tiles (26.05 and 26.01 ms a step at 128^3), slower elsewhere
  r.push_back(Sweep3D<2, 5, double, 32, 4, 2, 16, 16, 320, true, 2, false, 2>::entry());
  r.push_back(flex_sweep_entry<1, 5, 640>());
  r.push_back(flex_sweep_entry<2, 3, 512>());
  r.push_back(flex_sweep_entry<2, 1, 512>());
}

}  // namespace mfc
