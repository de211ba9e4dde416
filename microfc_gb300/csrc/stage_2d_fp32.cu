// Instantiations of the fused stage kernel for 2-D cases, split precision:
// FP32 WENO and HLLC, FP64 state, pressure recovery and RK update.
#include "mfc_launch.h"

namespace mfc {

// T x T tiles, interior ones loaded by TMA: 16x16 with 256 threads, four
// blocks per SM; 8x8 with 160, six blocks.
template <int NF, int T, bool GATE>
struct Pair2D {
  static StageEntry entry() {
    if constexpr (T == 16) return pair_entry<2, NF, 16, 16, 256, 4, 9, 9, GATE, false, true>();
    else return pair_entry<2, NF, 8, 8, 160, 6, 2, 2, GATE, false, true>();
  }
};

void register_stage_2d_fp32(std::vector<StageEntry>& r) {
  // the default; the autotuner may take either size alone
  r.push_back(sized_entry(Pair2D<2, 8, false>{}, Pair2D<2, 16, false>{}));
  r.push_back(Pair2D<2, 16, false>::entry());
  r.push_back(Pair2D<2, 8, false>::entry());
  r.push_back(pair_entry<2, 2, 16, 16, 256, 4, 9, 9>());
  r.push_back(sized_entry(Pair2D<1, 8, false>{}, Pair2D<1, 16, false>{}));
  r.push_back(stage_entry<2, 2, 3, float, 32, 16, 256>());
  r.push_back(stage_entry<2, 2, 1, float, 32, 16, 256>());
  r.push_back(stage_entry<2, 1, 3, float, 32, 16, 256>());
  r.push_back(stage_entry<2, 1, 1, float, 32, 16, 256>());
  // split precision with the learned WENO gate
  r.push_back(sized_entry(Pair2D<2, 8, true>{}, Pair2D<2, 16, true>{}));
  r.push_back(Pair2D<2, 16, true>::entry());
  r.push_back(Pair2D<2, 8, true>::entry());
  r.push_back(pair_entry<2, 2, 16, 16, 256, 4, 9, 9, true>());
  r.push_back(Pair2D<1, 16, true>::entry());
}

}  // namespace mfc
