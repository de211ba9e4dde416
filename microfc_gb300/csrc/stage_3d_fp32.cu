// Instantiations of the 3-D directional sweeps, split precision.
#include "mfc_launch.h"

namespace mfc {

void register_stage_3d_fp32(std::vector<StageEntry>& r) {
  // default: tiles staged by TMA bulk tensor copies; WENO5's y and z sweeps
  // run on pairs, seven blocks on an SM (256^3: 4987 us a step; five 5111,
  // uncapped 5234)
  r.push_back(Sweep3D<2, 5, float, 32, 4, 2, 16, 16, 256, true, 7, false, 7>::entry());
  r.push_back(Sweep3D<2, 5, float, 32, 4, 2, 16, 16, 256, false, 7, false, 7>::entry());
  r.push_back(Sweep3D<1, 5, float, 32, 4, 2, 16, 16, 256>::entry());
  r.push_back(Sweep3D<2, 3, float, 32, 4, 2, 16, 32, 256>::entry());
  r.push_back(Sweep3D<2, 1, float, 32, 4, 2, 16, 32, 256>::entry());
}

}  // namespace mfc
