// Instantiations of the 3-D directional sweeps, split precision.
#include "mfc_launch.h"

namespace mfc {

void register_stage_3d_fp32(std::vector<StageEntry>& r) {
  // (the plain-load form, 5414 us a step at 256^3 against 4799, is what the bulk
  // copies are compared with)
  r.push_back(PairSweep3D<2, 16, 128, 9, true, 7>::entry());
  r.push_back(PairSweep3D<2, 16, 128, 9, false, 7>::entry());
  r.push_back(PairSweep3D<1, 16, 128, 9, true, 7>::entry());
  r.push_back(Sweep3D<2, 3, float, 32, 4, 2, 16, 32, 256>::entry());
  r.push_back(Sweep3D<2, 1, float, 32, 4, 2, 16, 32, 256>::entry());
}

}  // namespace mfc
