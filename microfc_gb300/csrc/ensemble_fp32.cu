// Instantiations of the ensemble stage kernel, split precision.
#include "mfc_ensemble.cuh"

namespace mfc {

void register_ensemble_fp32(std::vector<EnsembleEntry>& r) {
  // interior tiles loaded by one TMA bulk tensor copy; the first is the default
  r.push_back(ensemble_entry<2, float, 16, 16, 256, 4, 9, 9, false, true>());
  r.push_back(ensemble_entry<2, float, 16, 16, 256, 4, 9, 9>());
  // with the viscous terms (mfc_gpu_ensemble_set_viscosity)
  r.push_back(ensemble_entry<2, float, 16, 16, 288, 3, 9, 9, false, true, true>());
}

void register_ensemble_gated(std::vector<EnsembleEntry>& r) {
  // interior tiles loaded by one TMA bulk tensor copy; the first is the default
  r.push_back(ensemble_entry<2, float, 16, 16, 256, 4, 9, 9, true, true>());
  r.push_back(ensemble_entry<2, float, 16, 16, 256, 4, 9, 9, true>());
  r.push_back(ensemble_entry<2, float, 16, 16, 256, 3, 9, 9, true, true>());
  // with the viscous terms (mfc_gpu_ensemble_set_viscosity)
  r.push_back(ensemble_entry<2, float, 16, 16, 288, 3, 9, 9, true, true, true>());
}

}  // namespace mfc
