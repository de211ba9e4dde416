// Instantiations of the 3-D directional sweeps, split precision.
#include "mfc_launch.h"

namespace mfc {

namespace {
// Blocks of 128 threads, seven on an SM; 384, whose threads take runs of three
// cells in place of nine, where the tiles of a sweep do not outnumber the SMs
// and a block has its SM for itself.  Where the line lies (us a step, 128 and
// 384 threads; before, 256): 26^3 (104 tiles) 51.6 and 34.7 (49.9), 32^3 (128)
// 51.9 and 34.1 (51.5), 40^3 (360) 65.4 and 57.5 (70.7), 56^3 95.8 and 98.6,
// 64^3 101.7 and 114.1 (123.6), 96^3 293 and 354.
template <int NF>
StageEntry sized_pairs() {
  using Few = PairSweep3D<NF, 16, 384, 3, true, 2>;
  using Many = PairSweep3D<NF, 16, 128, 9, true, 7>;
  struct Pick {
    static bool few(const int* n) {
      const int64_t x = (n[0] + 15) / 16, y = (n[1] + 15) / 16, z = (n[2] + 15) / 16;
      return x * y * n[2] <= flex::kSMs && x * z * n[1] <= flex::kSMs;
    }
  };
  StageEntry e = Many::entry();
  e.prepare = [] {
    const cudaError_t r = Few::prepare();
    return r == cudaSuccess ? Many::prepare() : r;
  };
  e.launch = [](const DevParams& P, const UniformCoef& U, const double* qin, const double* qbase, double* qout,
                double dt, int kind, cudaStream_t st) {
    return (Pick::few(P.n) ? &Few::launch : &Many::launch)(P, U, qin, qbase, qout, dt, kind, st);
  };
  e.launch_prims = [](const DevParams& P, const UniformCoef& U, const double* qin, const double* qbase, double* qout,
                      double dt, int kind, const PrimPairs& B, cudaStream_t st) {
    return (Pick::few(P.n) ? &Few::launch_prims : &Many::launch_prims)(P, U, qin, qbase, qout, dt, kind, B, st);
  };
  e.tile = [](const int* n, int* tx, int* ty, int* nt) {
    const StageEntry c = Pick::few(n) ? Few::entry() : Many::entry();
    *tx = c.tx;
    *ty = c.ty;
    *nt = c.nt;
  };
  return e;
}
}  // namespace

void register_stage_3d_fp32(std::vector<StageEntry>& r) {
  // (the plain-load form, 5414 us a step at 256^3 against 4799: the tests
  // compare the bulk copies' results with its own)
  r.push_back(sized_pairs<2>());
  r.push_back(PairSweep3D<2, 16, 128, 9, false, 7>::entry());
  r.push_back(sized_pairs<1>());
  r.push_back(Sweep3D<2, 3, float, 32, 4, 2, 16, 32, 256>::entry());
  r.push_back(Sweep3D<2, 1, float, 32, 4, 2, 16, 32, 256>::entry());
}

}  // namespace mfc
