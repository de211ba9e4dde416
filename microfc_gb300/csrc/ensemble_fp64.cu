// Instantiations of the ensemble stage kernel, FP64 (bit-faithful) arithmetic.
#include "mfc_ensemble.cuh"

namespace mfc {

void register_ensemble_fp64(std::vector<EnsembleEntry>& r) {
  r.push_back(ensemble_entry<2, double, 16, 16, 256, 1>());
  r.push_back(ensemble_entry<2, double, 32, 16, 512, 1>());
  r.push_back(ensemble_entry<2, double, 32, 8, 256, 1>());
  // with the viscous terms (mfc_gpu_ensemble_set_viscosity)
  r.push_back(ensemble_entry<2, double, 16, 16, 256, 1, 1, 1, false, false, true>());
  r.push_back(ensemble_entry<2, double, 32, 16, 512, 1, 1, 1, false, false, true>());
}

}  // namespace mfc
