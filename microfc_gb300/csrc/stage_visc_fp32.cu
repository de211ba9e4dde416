// Instantiations of the fused stage kernel with the viscous terms, split
// precision (FP32 reconstruction, Riemann and viscous fluxes; FP64 state):
// 1-D and 2-D, WENO5.
#include "mfc_launch.h"

namespace mfc {

// 16x16 tiles with 288 threads: the 544 faces of a tile, whose viscous fluxes
// are the longest phase, take two passes instead of three (214 us a step at
// 1024x512 against 254 with 256 threads at three blocks per SM, 233 at four).
template <int NF, int T>
struct Visc2D {
  static StageEntry entry() {
    if constexpr (T == 16) return pair_entry<2, NF, 16, 16, 288, 3, 9, 9, false, true, true>();
    else return pair_entry<2, NF, 8, 8, 160, 4, 2, 2, false, true, true>();
  }
};

void register_stage_visc_fp32(std::vector<StageEntry>& r) {
  r.push_back(pair_entry<1, 1, 62, 1, 96, 8, 2, 1, false, true>());
  r.push_back(pair_entry<1, 2, 62, 1, 96, 8, 2, 1, false, true>());
  r.push_back(sized_entry(Visc2D<1, 8>{}, Visc2D<1, 16>{}));
  r.push_back(sized_entry(Visc2D<2, 8>{}, Visc2D<2, 16>{}));
  r.push_back(Visc2D<2, 16>::entry());
  r.push_back(Visc2D<2, 8>::entry());
  // with the learned WENO gate (the gate chooses the weights; the viscous
  // fluxes are those of the split path)
  r.push_back(pair_entry<2, 2, 16, 16, 288, 3, 9, 9, true, true, true>());
  r.push_back(pair_entry<2, 1, 16, 16, 288, 3, 9, 9, true, true, true>());
}

}  // namespace mfc
