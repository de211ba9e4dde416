// Instantiations of the 3-D directional sweeps, FP64 arithmetic.
#include "mfc_launch.h"

namespace mfc {

namespace {
// Fixed tiles, TMA-staged: ahead of the sized ones where whole tiles cover the
// grid and there are enough waves of them (us a step, sized and fixed: 2.5
// waves, 64x64x48, 2756 and 2887; 3.4, 64^3, 3763 and 3380; 5.1, 96x64x64, 5132
// and 5248; 6.3, 96x80x64, 6562 and 6196; 7.6, 96x96x64, 7818 and 7590; 8.4,
// 160x64x64, 8705 and 8084; 11.4, 96^3, 11472 and 10894; 26.9, 128^3, 26540 and
// 25407; 256^3 205498 and 201893; where whole ones do not, 97x80x71 7477 and
// 8677, 60^3 2760 and 3216).  Both give the same bits.
using Fixed = Sweep3D<2, 5, double, 32, 4, 2, 16, 16, 320, true, 2, false, 2>;

bool whole_tiles(const int* n) {
  const int64_t tiles = (int64_t)(n[0] / 16) * (n[1] / 16) * n[2];  // of the y sweep, two on an SM
  return n[0] % 32 == 0 && n[1] % 16 == 0 && n[2] % 16 == 0 && tiles >= 6 * 2 * flex::kSMs;
}

StageEntry sized_or_fixed() {
  StageEntry e = flex_sweep_entry<2, 5, 640>();
  e.prepare = [] {
    const cudaError_t r = flex_sweep_entry<2, 5, 640>().prepare();
    return r == cudaSuccess ? Fixed::prepare() : r;
  };
  e.launch = [](const DevParams& P, const UniformCoef& U, const double* qin, const double* qbase, double* qout,
                double dt, int kind, cudaStream_t st) {
    return (whole_tiles(P.n) ? &Fixed::launch : flex_sweep_entry<2, 5, 640>().launch)(P, U, qin, qbase, qout, dt, kind,
                                                                                   st);
  };
  e.tile = [](const int* n, int* tx, int* ty, int* nt) {
    const StageEntry f = Fixed::entry();
    if (whole_tiles(n)) *tx = f.tx, *ty = f.ty, *nt = f.nt;
    else flex_sweep_entry<2, 5, 640>().tile(n, tx, ty, nt);
  };
  return e;
}
}  // namespace

void register_stage_3d_fp64(std::vector<StageEntry>& r) {
  r.push_back(sized_or_fixed());
  r.push_back(Fixed::entry());
  r.push_back(flex_sweep_entry<1, 5, 640>());
  r.push_back(flex_sweep_entry<2, 3, 512>());
  r.push_back(flex_sweep_entry<2, 1, 512>());
}

}  // namespace mfc
