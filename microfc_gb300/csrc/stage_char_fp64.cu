// Instantiations of the fused stage kernel that reconstructs the
// characteristic fields instead of the primitive variables (FP64, inviscid,
// WENO3/5; the fused kernel in 1-D and 2-D, the directional sweeps in 3-D;
// mfc_gpu_set_reconstruction).  The first entry per
// configuration is the default.
#include "mfc_launch.h"

namespace mfc {

namespace {
// 3-D: uncapped, the x sweep takes 128 registers, two blocks on an SM; with
// one block's budget 206, faster where the sweep's tiles do not outnumber the
// SMs (us a step, uncapped and capped; before, 179: 26^3 1090 and 945 (1034),
// 32^3 1102 and 948 (1035), 40^3 2620 and 2775 (3032), 128^3 45130 and 50080
// (53640)).
using Many = Sweep3D<2, 5, double, 32, 4, 2, 16, 16, 256, false, 0, true>;
using Few = Sweep3D<2, 5, double, 32, 4, 2, 16, 16, 256, false, 1, true, 1>;

StageEntry sized_sweeps() {
  StageEntry e = Many::entry();
  e.prepare = [] {
    const cudaError_t r = Few::prepare();
    return r == cudaSuccess ? Many::prepare() : r;
  };
  e.launch = [](const DevParams& P, const UniformCoef& U, const double* qin, const double* qbase, double* qout,
                double dt, int kind, cudaStream_t st) {
    const int64_t tiles = (int64_t)((P.n[0] + 31) / 32) * ((P.n[1] + 3) / 4) * ((P.n[2] + 1) / 2);
    return (tiles <= flex::kSMs ? &Few::launch : &Many::launch)(P, U, qin, qbase, qout, dt, kind, st);
  };
  return e;
}
}  // namespace

void register_stage_char_fp64(std::vector<StageEntry>& r) {
#define MFC_CHAR(ND, NF, WO, TX, TY, NT) \
  r.push_back(stage_entry<ND, NF, WO, double, TX, TY, NT, false, false, true>());
  MFC_CHAR(2, 2, 5, 32, 16, 512)
  MFC_CHAR(2, 2, 5, 16, 16, 256)
  MFC_CHAR(2, 1, 5, 32, 16, 512)
  MFC_CHAR(2, 2, 3, 16, 16, 256)
  MFC_CHAR(2, 1, 3, 16, 16, 256)
  MFC_CHAR(1, 2, 5, 128, 1, 128)
  MFC_CHAR(1, 1, 5, 128, 1, 128)
  MFC_CHAR(1, 2, 3, 128, 1, 128)
  MFC_CHAR(1, 1, 3, 128, 1, 128)
#undef MFC_CHAR
  // 3-D: the directional sweeps
  r.push_back(sized_sweeps());
  r.push_back(Sweep3D<1, 5, double, 32, 4, 2, 16, 16, 256, false, 0, true>::entry());
  r.push_back(Sweep3D<2, 3, double, 32, 4, 2, 16, 16, 256, false, 0, true>::entry());
}

}  // namespace mfc
