// Instantiations of the ensemble stage kernel, FP64 (bit-faithful) arithmetic.
#include "mfc_ensemble.cuh"

namespace mfc {

// The 256-thread tiles cap their registers at 128 so that two blocks share an
// SM (uncapped, 150 registers and one block: 24 droplets of 128x64 to 512x256
// 14.8 ms a step against 11.5, viscous 20.1 against 15.0; persistent blocks
// before 13.5 and 17.7).
void register_ensemble_fp64(std::vector<EnsembleEntry>& r) {
  r.push_back(ensemble_entry<2, double, 16, 16, 256, 2>());
  r.push_back(ensemble_entry<2, double, 32, 16, 512, 1>());
  r.push_back(ensemble_entry<2, double, 32, 8, 256, 2>());
  // with the viscous terms (mfc_gpu_ensemble_set_viscosity)
  r.push_back(ensemble_entry<2, double, 16, 16, 256, 2, 1, 1, false, false, true>());
  r.push_back(ensemble_entry<2, double, 32, 16, 512, 1, 1, 1, false, false, true>());
}

}  // namespace mfc
