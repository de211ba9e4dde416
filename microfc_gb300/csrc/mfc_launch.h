// Internal launcher registry: every compiled instantiation of the stage
// kernel registers one entry; the C ABI picks the entry matching the case's
// dimensionality, fluid count, WENO order, precision and tile variant.
#pragma once

#include <cuda_runtime.h>

#include <string>
#include <vector>

#include <type_traits>
#include <utility>

#include "../../include/mfc_gpu.h"
#include "mfc_device.cuh"
#include "mfc_flex.cuh"
#include "mfc_pair.cuh"
#include "mfc_stage.cuh"
#include "mfc_pair_sweep.cuh"
#include "mfc_sweep.cuh"

namespace mfc {

struct StageEntry {
  int nd, nf, wo, prec;  // prec: an MFC_PREC_* value
  int tx, ty, nt;
  size_t smem;
  int kernels;  // kernel launches per RK stage (1 in 1-D/2-D, 3 sweeps in 3-D)
  cudaError_t (*prepare)();
  cudaError_t (*launch)(const DevParams& P, const UniformCoef& U, const double* qin, const double* qbase,
                        double* qout, double dt, int kind, cudaStream_t st);
  bool visc = false;  // compiled with the viscous terms
  bool tma = false;   // interior tiles staged by a TMA bulk tensor copy
  bool chr = false;   // WENO of the characteristic fields (MFC_RECON_CHARACTERISTIC)
  // the same launch with primitive pairs (mfc_pair.cuh); null: the kernel has no use for them
  cudaError_t (*launch_prims)(const DevParams& P, const UniformCoef& U, const double* qin, const double* qbase,
                              double* qout, double dt, int kind, const PrimPairs& B, cudaStream_t st) = nullptr;
  // the tile and threads of a grid of n[0] x n[1] x n[2] cells where the launch chooses them (else tx, ty, nt)
  void (*tile)(const int* n, int* tx, int* ty, int* nt) = nullptr;
};

// Launches a stage kernel with programmatic stream serialization, so that
// it may become resident while the previous kernel on the stream drains
// (the kernel waits for that kernel's results with griddep_wait).
template <class... KArgs, class... Args>
cudaError_t launch_dependent(void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t st,
                             Args&&... args) {
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kernel, std::forward<Args>(args)...);
}

// TMA selects the kernel that stages interior tiles with a bulk tensor copy;
// FMA the instantiations compiled with multiply-add contraction
// (MFC_PREC_FP64_FMA); CHAR WENO of the characteristic fields.
template <int ND, int NF, int WO, class RT, int TX, int TY, int NT, bool TMA = false, bool FMA = false,
          bool CHAR = false>
StageEntry stage_entry() {
  static_assert(!FMA || sizeof(RT) == 8, "the contracted variant is FP64");
  static_assert(!TMA || (ND == 2 && !CHAR), "TMA staging is compiled for the inviscid 2-D kernel");
  struct K {
    static constexpr auto func() {
      if constexpr (TMA) return &stage_kernel_tma<ND, NF, WO, RT, TX, TY, NT, FMA>;
      else return &stage_kernel<ND, NF, WO, RT, TX, TY, NT, FMA, CHAR>;
    }
    static constexpr size_t smem() { return stage_smem_total<ND, NF, WO, RT, TX, TY, false, TMA>(); }
  };
  StageEntry e{};
  e.nd = ND;
  e.nf = NF;
  e.wo = WO;
  e.prec = FMA ? MFC_PREC_FP64_FMA : sizeof(RT) == 8 ? MFC_PREC_FP64 : MFC_PREC_SPLIT;
  e.tx = TX;
  e.ty = TY;
  e.nt = NT;
  e.smem = K::smem();
  e.kernels = 1;
  e.prepare = [] {
    return cudaFuncSetAttribute(K::func(), cudaFuncAttributeMaxDynamicSharedMemorySize, (int)K::smem());
  };
  e.launch = [](const DevParams& P, const UniformCoef&, const double* qin, const double* qbase, double* qout,
                double dt, int kind, cudaStream_t st) {
    const dim3 grid((unsigned)((P.n[0] + TX - 1) / TX), ND > 1 ? (unsigned)((P.n[1] + TY - 1) / TY) : 1u);
    if constexpr (TMA) {
      // the map of this launch's input register; without one (a layout the
      // copy engine does not take) every tile takes the plain loads
      using Sh = StageShape<ND, NF, WO, RT, TX, TY>;
      TileMap T{};
      encode_tile_map(T, qin, P.n[0], P.n[1], Sh::S, P.sy, P.sv, TmaBox<TX, Sh::H>::kWidth, Sh::LY);
      return launch_dependent(K::func(), grid, dim3(NT), K::smem(), st, P, T, qin, qbase, qout, dt, kind);
    } else {
      return launch_dependent(K::func(), grid, dim3(NT), K::smem(), st, P, qin, qbase, qout, dt, kind);
    }
  };
  e.tma = TMA;
  e.chr = CHAR;
  return e;
}

// The split WENO5 kernels of 1-D and 2-D cases (mfc_pair.cuh).
template <int ND, int NF, int TX, int TY, int NT, int MINB, int RX, int RY, bool GATE = false, bool VISC = false,
          bool TMA = false>
StageEntry pair_entry() {
  static_assert(!TMA || ND == 2, "TMA loads are compiled for the 2-D kernel");
  struct K {
    static constexpr auto func() {
      if constexpr (TMA) return &pair_kernel_tma<NF, TX, TY, NT, GATE, VISC, MINB, RX, RY>;
      else return &pair_kernel<ND, NF, TX, TY, NT, GATE, VISC, MINB, RX, RY>;
    }
  };
  StageEntry e{};
  e.nd = ND;
  e.nf = NF;
  e.wo = 5;
  e.prec = GATE ? MFC_PREC_GATED : MFC_PREC_SPLIT;
  e.tx = TX;
  e.ty = TY;
  e.nt = NT;
  e.smem = pair_smem<ND, NF, TX, TY, NT, GATE, VISC, TMA>(false);
  e.kernels = 1;
  e.prepare = [] {
    return cudaFuncSetAttribute(K::func(), cudaFuncAttributeMaxDynamicSharedMemorySize,
                                (int)pair_smem<ND, NF, TX, TY, NT, GATE, VISC, TMA>(false));
  };
  e.launch_prims = [](const DevParams& P, const UniformCoef& U, const double* qin, const double* qbase, double* qout,
                      double dt, int kind, const PrimPairs& B, cudaStream_t st) {
    const dim3 grid((unsigned)((P.n[0] + TX - 1) / TX), ND > 1 ? (unsigned)((P.n[1] + TY - 1) / TY) : 1u);
    // a uniform grid stages no coefficient records: launch without their share
    const size_t smem = pair_smem<ND, NF, TX, TY, NT, GATE, VISC, TMA>(U.on[0] && (ND < 2 || U.on[1]));
    if constexpr (TMA) {
      // the map of this launch's input; without one (a layout the copy engine
      // does not take) every tile takes the plain loads
      using Sh = PairShape<ND, NF, TX, TY, VISC>;
      TileMap T{};
      if (B.in != nullptr)
        encode_tile_map(T, reinterpret_cast<const double*>(B.in), (int)B.pitch, P.n[1], Sh::NPR, B.pitch, B.plane,
                        Sh::LX, Sh::LY);
      else
        encode_tile_map(T, qin, P.n[0], P.n[1], Sh::S, P.sy, P.sv, TmaBox<TX, Sh::H>::kWidth, Sh::LY);
      return launch_dependent(K::func(), grid, dim3(NT), smem, st, P, U, T, qin, qbase, qout, dt, kind, B);
    } else {
      return launch_dependent(K::func(), grid, dim3(NT), smem, st, P, U, qin, qbase, qout, dt, kind, B);
    }
  };
  e.launch = [](const DevParams& P, const UniformCoef& U, const double* qin, const double* qbase, double* qout,
                double dt, int kind, cudaStream_t st) {
    return pair_entry<ND, NF, TX, TY, NT, MINB, RX, RY, GATE, VISC, TMA>().launch_prims(P, U, qin, qbase, qout, dt, kind,
                                                                                        PrimPairs{}, st);
  };
  e.visc = VISC;
  e.tma = TMA;
  return e;
}

// Two pair entries as one: tiles of 8x8 cells where 16x16 ones are too few
// to fill the chip (kSmallTiles of them or less: up to there the 8x8 ones, six
// blocks on an SM, are one wave), else 16x16.  Where the line lies (us a step,
// 8x8 and 16x16, two fluids): 100x50 (28 tiles) split 13.7 and 19.1, gated 17.0
// and 26.2, viscous 20.7 and 25.2; 333x167 (231) split 22.3 and 27.9, one fluid
// 20.3 and 23.1, gated 25.9 and 31.9, viscous 33.1 and 36.1, weno_Re_flux 67.7
// and 69.5; 360x180 (276) split 29.2 and 30.0, stretched 32.9 and 29.9, one
// fluid 25.3 and 24.3, gated 35.5 and 34.2, viscous 44.3 and 37.9,
// weno_Re_flux 80.5 and 71.3; 512x256 (512) split 45.4 and 37.0.
constexpr int64_t kSmallTiles = 240;
template <class Small, class Large>
StageEntry sized_entry(const Small&, const Large&) {
  StageEntry e = Large::entry();
  e.prepare = [] {
    const cudaError_t r = Small::entry().prepare();
    return r != cudaSuccess ? r : Large::entry().prepare();
  };
  struct Pick {
    static bool small(const int* n) {
      return (int64_t)((n[0] + 15) / 16) * ((n[1] + 15) / 16) <= kSmallTiles;
    }
  };
  e.launch = [](const DevParams& P, const UniformCoef& U, const double* qin, const double* qbase, double* qout,
                double dt, int kind, cudaStream_t st) {
    return (Pick::small(P.n) ? Small::entry() : Large::entry()).launch(P, U, qin, qbase, qout, dt, kind, st);
  };
  e.launch_prims = [](const DevParams& P, const UniformCoef& U, const double* qin, const double* qbase, double* qout,
                      double dt, int kind, const PrimPairs& B, cudaStream_t st) {
    return (Pick::small(P.n) ? Small::entry() : Large::entry()).launch_prims(P, U, qin, qbase, qout, dt, kind, B, st);
  };
  e.tile = [](const int* n, int* tx, int* ty, int* nt) {
    const StageEntry c = Pick::small(n) ? Small::entry() : Large::entry();
    *tx = c.tx;
    *ty = c.ty;
    *nt = c.nt;
  };
  return e;
}

// Tile sizes of the flex kernels: the ones with the least work on the
// busiest SM, ceil(tiles / 152) tiles of the largest size.  A tile's cost in
// SM cycles, from the operation counts of the formulas and the FP64 unit's
// measured rates: a phase takes 16.5 cycles per warp operation once four
// warps are busy, but at least 64 per operation of one warp's chain of items;
// loads, barriers and the block's launch take about 8000 more.  Candidates:
// the smallest tile of each number of columns and rows that fits shared
// memory.  A plan is a pure function of the sizes; each thread remembers
// those of the last few grids (a search takes about 0.1 ms).
namespace flex {
constexpr int kSMs = 152;
constexpr double kRate = 16.5, kChain = 64.0, kTile = 8000.0;
constexpr double weno_ops(int wo) { return wo == 5 ? 72 : wo == 3 ? 26 : 0; }
constexpr double weno_side_ops(int wo) { return wo == 5 ? 53 : wo == 3 ? 18 : 0; }
inline int groups(int n) { return (n + 31) / 32; }
// a phase of `ops` warp operations in g groups of at most `item` operations
inline double phase(double ops, int g, double item, int warps) {
  const double chain = kChain * item * ((g + warps - 1) / warps);
  return ops * kRate > chain ? ops * kRate : chain;
}

// The sizes (x, y) that minimise ceil(tiles / 152) * cost(x, y) over grids
// of nx x ny x layers cells cut into ceil(nx / x) * ceil(ny / y) * layers
// tiles, with lo <= x <= hi_x, y <= hi_y and fits(x, y).
struct Plan {
  int key[3] = {0, 0, 0}, x = 0, y = 0;
};
template <class Cost, class Fits>
Plan search(int nx, int ny, int layers, int lo_x, int hi_x, int lo_y, int hi_y, Cost&& cost, Fits&& fits) {
  Plan best{{nx, ny, layers}, 1, 1};
  double least = 0.0;
  lo_x = lo_x < nx ? lo_x : nx;
  lo_y = lo_y < ny ? lo_y : ny;
  for (int c = 1, last_x = 0; c <= nx; ++c) {
    const int x = (nx + c - 1) / c;
    if (x == last_x || x > hi_x) continue;
    last_x = x;
    if (x < lo_x) break;
    for (int r = 1, last_y = 0; r <= ny; ++r) {
      const int y = (ny + r - 1) / r;
      if (y == last_y || y > hi_y) continue;
      last_y = y;
      if (y < lo_y) break;
      if (!fits(x, y)) continue;
      const int64_t tiles = (int64_t)((nx + x - 1) / x) * ((ny + y - 1) / y) * layers;
      const double t = double((tiles + kSMs - 1) / kSMs) * cost(x, y);
      if (least == 0.0 || t < least) {
        least = t;
        best.x = x;
        best.y = y;
      }
    }
  }
  return best;
}
// The remembered plan of a grid, or a new search.
template <class Search>
Plan remembered(Plan (&memo)[8], unsigned& next, int nx, int ny, int layers, Search&& s) {
  for (const Plan& m : memo)
    if (m.key[0] == nx && m.key[1] == ny && m.key[2] == layers) return m;
  return memo[next++ % 8] = s();
}

template <int ND, int NF, int WO, int NT, bool VISC>
Plan plan(int nx, int ny) {
  using Sh = FlexShape<ND, NF, WO>;
  thread_local Plan memo[8];
  thread_local unsigned next = 0;
  return remembered(memo, next, nx, ny, 1, [&] {
    constexpr int S = Sh::S, H = Sh::H, NW = NT / 32;
    constexpr double both = weno_ops(WO), one = weno_side_ops(WO);
    constexpr double face = VISC ? 150 : 85, prim = 14, cell = ND > 1 ? 14 : 9;
    auto cost = [&](int x, int y) {
      const int gi = groups(S * x * y), ge = groups(S * y) + (ND > 1 ? groups(S * x) : 0);
      const int gf = groups((x + 1) * y) + (ND > 1 ? groups(x * (y + 1)) : 0);
      const int gl = groups(x * y + 2 * H * (y + (ND > 1 ? x : 0)));
      double weno = phase(ND * gi * both + 2 * ge * one, ND * gi + 2 * ge, both, NW), hllc = phase(gf * face, gf, face, NW);
      if (ND == 1) {
        const int gs = groups(S * (x + 1)), gp = groups(2 * (x + 1));
        if (flex_sides<WO>(gi, ge, gs, NW)) weno = phase(2 * gs * one, 2 * gs, one, NW);
        if (!VISC && flex_lane_pairs(x + 1, NW)) hllc = phase(gp * 59.0, gp, 59.0, NW);
      }
      return phase(gl * prim, gl, prim, NW) + weno + hllc + phase(gi * cell, gi, cell, NW) + kTile;
    };
    // (a launch takes 65535 rows of tiles)
    return search(nx, ny, 1, ND > 1 ? 4 : 2, ND > 1 ? 96 : 512, ND > 1 ? 4 : 1, 96, cost, [ny](int x, int y) {
      return Sh::bytes(x, y) <= kFlexSmemMax && (ny + y - 1) / y <= 65535;
    });
  });
}

// x: cells along the sweep, y: pencils
template <int NF, int WO, int NT, int DIR>
Plan sweep_plan(int na, int nb, int nc) {
  using Sh = FlexSweepShape<NF, WO, DIR>;
  thread_local Plan memo[8];
  thread_local unsigned next = 0;
  return remembered(memo, next, na, nb, nc, [&] {
    constexpr int S = Sh::S, H = Sh::H, NW = NT / 32;
    constexpr double both = weno_ops(WO), one = weno_side_ops(WO);
    constexpr double face = 90, prim = DIR == 0 ? 17 : 0, cell = DIR == 2 ? 10 : 4;
    auto cost = [&](int a, int p) {
      const int gi = groups(S * a * p), ge = groups(S * p), gf = groups((a + 1) * p), gl = groups((a + 2 * H) * p);
      return phase(gl * prim, gl, prim, NW) + phase(gi * both + 2 * ge * one, gi + 2 * ge, both, NW) +
             phase(gf * face, gf, face, NW) + phase(gi * cell, gi, cell, NW) + kTile;
    };
    // y and z: at least eight pencils, one 64-byte line of x per row
    return search(na, nb, nc, 4, 512, DIR == 0 ? 1 : 8, 256, cost, [](int a, int p) { return Sh::bytes(a, p) <= kFlexSmemMax; });
  });
}
}  // namespace flex

template <int ND, int NF, int WO, int NT, bool VISC = false>
StageEntry flex_entry() {
  StageEntry e{};
  e.nd = ND;
  e.nf = NF;
  e.wo = WO;
  e.prec = MFC_PREC_FP64;
  e.nt = NT;
  e.smem = kFlexSmemMax;
  e.kernels = 1;
  e.prepare = [] {
    return cudaFuncSetAttribute(&flex_kernel<ND, NF, WO, NT, VISC>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                (int)kFlexSmemMax);
  };
  e.launch = [](const DevParams& P, const UniformCoef&, const double* qin, const double* qbase, double* qout,
                double dt, int kind, cudaStream_t st) {
    const flex::Plan t = flex::plan<ND, NF, WO, NT, VISC>(P.n[0], P.n[1]);
    const dim3 grid((unsigned)((P.n[0] + t.x - 1) / t.x), (unsigned)((P.n[1] + t.y - 1) / t.y));
    return launch_dependent(&flex_kernel<ND, NF, WO, NT, VISC>, grid, dim3(NT), FlexShape<ND, NF, WO>::bytes(t.x, t.y),
                            st, P, qin, qbase, qout, dt, kind, t.x, t.y);
  };
  e.visc = VISC;
  e.tile = [](const int* n, int* tx, int* ty, int* nt) {
    const flex::Plan t = flex::plan<ND, NF, WO, NT, VISC>(n[0], n[1]);
    *tx = t.x;
    *ty = t.y;
    *nt = NT;
  };
  return e;
}

// 3-D: three flex sweeps per stage.
template <int NF, int WO, int NT>
StageEntry flex_sweep_entry() {
  StageEntry e{};
  e.nd = 3;
  e.nf = NF;
  e.wo = WO;
  e.prec = MFC_PREC_FP64;
  e.nt = NT;
  e.smem = kFlexSmemMax;
  e.kernels = 3;
  e.prepare = [] {
    const auto attr = cudaFuncAttributeMaxDynamicSharedMemorySize;
    cudaError_t r = cudaFuncSetAttribute(&flex_sweep_kernel<NF, WO, NT, 0>, attr, (int)kFlexSmemMax);
    if (r == cudaSuccess) r = cudaFuncSetAttribute(&flex_sweep_kernel<NF, WO, NT, 1>, attr, (int)kFlexSmemMax);
    if (r == cudaSuccess) r = cudaFuncSetAttribute(&flex_sweep_kernel<NF, WO, NT, 2>, attr, (int)kFlexSmemMax);
    return r;
  };
  e.launch = [](const DevParams& P, const UniformCoef&, const double* qin, const double* qbase, double* qout,
                double dt, int kind, cudaStream_t st) {
    auto sweep = [&](auto dir) {
      constexpr int D = decltype(dir)::value;
      constexpr int A = D, B = D == 0 ? 1 : 0, C = D == 2 ? 1 : 2;
      const flex::Plan t = flex::sweep_plan<NF, WO, NT, D>(P.n[A], P.n[B], P.n[C]);
      const unsigned tiles =
          (unsigned)((P.n[A] + t.x - 1) / t.x) * (unsigned)((P.n[B] + t.y - 1) / t.y) * (unsigned)P.n[C];
      return launch_dependent(&flex_sweep_kernel<NF, WO, NT, D>, dim3(tiles), dim3(NT),
                              FlexSweepShape<NF, WO, D>::bytes(t.x, t.y), st, P, qin, qbase, qout, dt, kind, t.x, t.y);
    };
    cudaError_t r = sweep(std::integral_constant<int, 0>{});
    if (r == cudaSuccess) r = sweep(std::integral_constant<int, 1>{});
    if (r == cudaSuccess) r = sweep(std::integral_constant<int, 2>{});
    return r;
  };
  e.tile = [](const int* n, int* tx, int* ty, int* nt) {  // the x sweep's
    const flex::Plan t = flex::sweep_plan<NF, WO, NT, 0>(n[0], n[1], n[2]);
    *tx = t.x;
    *ty = t.y;
    *nt = NT;
  };
  return e;
}

// 3-D: three directional sweeps per stage (mfc_sweep.cuh).  The x sweep uses
// TA0 x TB0 x TC0 tiles (x along the sweep); the y and z sweeps use
// TA1 x TB1 x 1 tiles with x across the pencils.  TMA: tiles whose sweep
// halo lies inside the domain arrive by one bulk tensor copy.
// MINB2 > 0 caps the registers of the z sweep (which also does the RK
// combination) so that MINB2 of its blocks fit on an SM; MINB01 does the same
// for the x and y sweeps.
template <int NF, int WO, class RT, int TA0, int TB0, int TC0, int TA1, int TB1, int NT, bool TMA = false,
          int MINB2 = 0, bool CHAR = false, int MINB01 = 0>
struct Sweep3D {
  template <int DIR>
  using K = std::conditional_t<DIR == 0, SweepShape<NF, WO, RT, 0, TA0, TB0, TC0>,
                               SweepShape<NF, WO, RT, DIR, TA1, TB1, 1>>;
  template <int DIR>
  static constexpr auto func() {
    if constexpr (DIR == 0) return &sweep_kernel<NF, WO, RT, 0, TA0, TB0, TC0, NT, TMA, MINB01, CHAR>;
    else if constexpr (DIR == 2) return &sweep_kernel<NF, WO, RT, 2, TA1, TB1, 1, NT, TMA, MINB2, CHAR>;
    else return &sweep_kernel<NF, WO, RT, DIR, TA1, TB1, 1, NT, TMA, MINB01, CHAR>;
  }

  template <int DIR>
  static cudaError_t prep() {
    return cudaFuncSetAttribute(func<DIR>(), cudaFuncAttributeMaxDynamicSharedMemorySize, (int)K<DIR>::kSmemBytes);
  }
  static cudaError_t prepare() {
    cudaError_t e = prep<0>();
    if (e == cudaSuccess) e = prep<1>();
    if (e == cudaSuccess) e = prep<2>();
    return e;
  }
  // the map of the sweep's box (none: plain loads): the stage input for the
  // x sweep, the primitives the x sweep stores (the work buffer's second
  // segment, reconstruction type) for the y and z sweeps
  template <int DIR>
  static TileMap tile_map(const DevParams& P, const double* qin) {
    TileMap T{};
    if constexpr (TMA && K<DIR>::kTmaFits) {
      constexpr int S = K<DIR>::S;
      const void* base = DIR == 0 ? static_cast<const void*>(qin)
                                  : static_cast<const void*>(static_cast<const RT*>(P.work) + int64_t(S) * P.sv);
      encode_tile_map_3d(T, base, K<DIR>::kStageElem, P.n[0], P.n[1], P.n[2], S, P.sy, P.sz, P.sv, K<DIR>::BX,
                         K<DIR>::BY, K<DIR>::BZ);
    }
    return T;
  }
  static cudaError_t launch(const DevParams& P, const UniformCoef& U, const double* qin, const double* qbase,
                            double* qout, double dt, int kind, cudaStream_t st) {
    const unsigned nx = P.n[0], ny = P.n[1], nz = P.n[2];
    const dim3 g0((nx + TA0 - 1) / TA0, (ny + TB0 - 1) / TB0, (nz + TC0 - 1) / TC0);
    const dim3 g1((nx + TB1 - 1) / TB1, (ny + TA1 - 1) / TA1, nz);
    const dim3 g2((nx + TB1 - 1) / TB1, (nz + TA1 - 1) / TA1, ny);
    const TileMap T0 = tile_map<0>(P, qin), T1 = tile_map<1>(P, qin), T2 = tile_map<2>(P, qin);
    cudaError_t e =
        launch_dependent(func<0>(), g0, dim3(NT), K<0>::kSmemBytes, st, P, T0, qin, qbase, qout, dt, kind);
    if (e == cudaSuccess)
      e = launch_dependent(func<1>(), g1, dim3(NT), K<1>::kSmemBytes, st, P, T1, qin, qbase, qout, dt, kind);
    if (e == cudaSuccess)
      e = launch_dependent(func<2>(), g2, dim3(NT), K<2>::kSmemBytes, st, P, T2, qin, qbase, qout, dt, kind);
    return e;
  }
  static StageEntry entry() {
    static_assert(!TMA || (K<0>::kTmaFits && K<1>::kTmaFits && K<2>::kTmaFits),
                  "the TMA box of every sweep must fit its WENO and flux arrays");
    return StageEntry{3, NF, WO, sizeof(RT) == 8 ? 0 : 1, TA0, TB1, NT, K<1>::kSmemBytes, 3, &prepare, &launch,
                      false, TMA, CHAR};
  }
};

// Split WENO5: the three sweeps on primitive pairs (mfc_pair_sweep.cuh), tiles
// of TA cells along the sweep and 16 pencils.  TMA: interior tiles by one
// bulk tensor copy.
template <int NF, int TA, int NT, int R, bool TMA, int MINB>
struct PairSweep3D {
  static constexpr int TB = 16;
  template <int DIR>
  using K = PairSweepShape<NF, DIR, TA, TB>;
  template <int DIR>
  static constexpr auto func() {
    return &pair_sweep_kernel<NF, DIR, TA, TB, NT, R, TMA, MINB>;
  }
  template <int DIR>
  static cudaError_t prep() {
    return cudaFuncSetAttribute(func<DIR>(), cudaFuncAttributeMaxDynamicSharedMemorySize,
                                (int)(K<DIR>::kCoefOffset + K<DIR>::kCoefBytes));
  }
  static cudaError_t prepare() {
    cudaError_t e = prep<0>();
    if (e == cudaSuccess) e = prep<1>();
    if (e == cudaSuccess) e = prep<2>();
    return e;
  }
  template <int DIR>
  static cudaError_t sweep(dim3 grid, const DevParams& P, const UniformCoef& U, const double* qin, const double* qbase,
                           double* qout, double dt, int kind, const PrimPairs& B, cudaStream_t st) {
    TileMap T{};
    if constexpr (TMA)  // 8-byte elements, a tile in its final layout
      encode_tile_map_3d(T, B.cur, 8, P.n[0], P.n[1], P.n[2], K<DIR>::NPR, P.sy, P.sz, P.sv,
                         DIR == 0 ? K<DIR>::PLA : TB, DIR == 0 ? TB : DIR == 1 ? K<DIR>::LA : 1,
                         DIR == 2 ? K<DIR>::LA : 1);
    return launch_dependent(func<DIR>(), grid, dim3(NT), K<DIR>::kCoefOffset + (U.on[DIR] ? 0 : K<DIR>::kCoefBytes), st,
                            P, U, T, qin, qbase, qout, dt, kind, B);
  }
  static cudaError_t launch_prims(const DevParams& P, const UniformCoef& U, const double* qin, const double* qbase,
                                  double* qout, double dt, int kind, const PrimPairs& B, cudaStream_t st) {
    const unsigned nx = P.n[0], ny = P.n[1], nz = P.n[2];
    auto tiles = [](unsigned n, unsigned t) { return (n + t - 1) / t; };
    cudaError_t e = sweep<0>(dim3(tiles(nx, TA), tiles(ny, TB), nz), P, U, qin, qbase, qout, dt, kind, B, st);
    if (e == cudaSuccess) e = sweep<1>(dim3(tiles(nx, TB), tiles(ny, TA), nz), P, U, qin, qbase, qout, dt, kind, B, st);
    if (e == cudaSuccess) e = sweep<2>(dim3(tiles(nx, TB), tiles(nz, TA), ny), P, U, qin, qbase, qout, dt, kind, B, st);
    return e;
  }
  static cudaError_t launch(const DevParams& P, const UniformCoef& U, const double* qin, const double* qbase,
                            double* qout, double dt, int kind, cudaStream_t st) {
    const PrimPairs B{nullptr, nullptr, 0, 0, reinterpret_cast<f32x2*>(P.work) + int64_t(K<0>::NPR) * P.sv};
    return launch_prims(P, U, qin, qbase, qout, dt, kind, B, st);
  }
  static StageEntry entry() {
    StageEntry e{3, NF, 5, 1, TA, TB, NT, K<0>::kCoefOffset + K<0>::kCoefBytes, 3, &prepare, &launch, false, TMA};
    e.launch_prims = &launch_prims;
    return e;
  }
};

// What the standalone entry points of other translation units need from a
// context (mfc_gpu_ctx is private to mfc_capi.cu).
struct CtxView {
  const DevParams* dev = nullptr;  // the context's kernel parameters
  const double* q0 = nullptr;      // register 0 (q_cons_ts(1))
  cudaStream_t stream = nullptr;
  int nd = 0, nf = 0, wo = 0, S = 0, prec = 0;
  int n[3] = {1, 1, 1};
  bool visc = false, has_proc = false;
  int64_t* launches = nullptr;     // the context's launch counter
};
bool ctx_view(mfc_gpu_ctx* c, CtxView& v);

// The context's device scratch, at least `bytes` long (grown on demand, freed
// with the context); for entry points that synchronise before returning.
cudaError_t ctx_scratch(mfc_gpu_ctx* c, size_t bytes, void** out);

// weno_Re_flux = T (mfc_visc_grad.cu): device buffers of the gradient
// preparation -- the velocities ([ND][ny+10][nx+10] from x = y = -5; one row
// in 1-D), the cell gradients ([ND*ND][ny+6][nx+6] from x = y = -3; one row
// in 1-D), the face gradients (ViscParams::fg), the cell widths of each
// direction for cells -kCoefPad .. n-1+kCoefPad and, for the split and gated
// precisions, an FP32 table per direction: the WENO coefficients of those
// cells ([kNumCoef][n + 2 kCoefPad]) followed by their inverse widths.
// In 2-D those precisions hold the velocities and the face gradients as FP32
// pairs of the two components (fg[0]: [d][ny][nx + 1]), and no cell gradients.
// uniform: their coefficients, then the inverse width, as (c, c) pairs, when
// every cell of each direction has the same.
struct GradCoef {
  int on = 0;
  unsigned long long rec[2][kCoefRec] = {};
};
struct ViscGradBuffers {
  GradCoef uniform;
  double* vel = nullptr;
  double* g = nullptr;
  double* fg[2] = {nullptr, nullptr};
  double* w[2] = {nullptr, nullptr};
  float* cf[2] = {nullptr, nullptr};
};
// Launches of one preparation: 3 in 1-D, 4 in 2-D, 2 in 2-D with fp32.
inline int visc_gradients_launches(int nd, bool fp32) { return nd == 1 ? 3 : fp32 ? 2 : 4; }
// Prepares the face gradients of the stage input q on stream st, reconstructing in FP32 when fp32 is set (split and
// gated contexts), else in FP64.
cudaError_t visc_gradients_launch(int nd, int nf, bool fp32, const DevParams& P, const ViscGradBuffers& B,
                                  const double* q, cudaStream_t st);

// The default (first registered) launcher of a configuration, or nullptr.
const StageEntry* find_stage(int nd, int nf, int wo, int prec, bool visc = false, bool chr = false);

// Records msg as the calling thread's mfc_gpu_last_error() and returns code.
int report_error(int code, const std::string& msg);

// Makes the pages of a host array that a device copy is about to fill resident
// and recently used.  On Grace a copy into fresh pages faults them in one by
// one from the GPU's side, about 40 us per 64 KB page: 24 fresh ensemble states
// (82 MB) took 52 ms to download, 4.4 ms with this.  And pages that the CPU has
// not used for a while cost a copy 2 to 3 us each now and then, pinned ones too:
// of 180 downloads of a pinned 1.07 GB state 26 took 40 to 100 ms instead of
// 5.6, of as many with a read of each page (5.9 ms) one to three.
//
// Pinned arrays: one read per page.  Pageable ones of up to 256 pages: one
// store, which the copy overwrites.  Larger ones: the kernel is asked to
// populate the range where pages of the middle are missing, else one read per
// page.  Other addresses are left alone.  (us a download, without, with: 112 KB
// fresh 104 and 27, again into the same array 12.3 and 12.6, pinned 11.7 and
// 11.7; 28 MB fresh 1230 and 1075, again 164.8 and 172.7, pinned 163.5 and 168.6.)
void populate_pages(void* p, size_t bytes);

// Gate training samples of a 2-D state (mfc_gate.cu).
int gate_samples(const DevParams& P, int nf, const double* q, int dir, float* xout, float* dev_out, cudaStream_t st);

// FP32 gate parameters (host) -> FP16 device copy (mfc_gate.cu).
int gate_upload(const float* host_params, void* dev_half, cudaStream_t st);

// Defined in the instantiation translation units.
void register_stage_1d_fp64(std::vector<StageEntry>& r);
void register_stage_1d_fp32(std::vector<StageEntry>& r);
void register_stage_2d_fp64(std::vector<StageEntry>& r);
void register_stage_2d_fp64fma(std::vector<StageEntry>& r);
void register_stage_2d_fp32(std::vector<StageEntry>& r);
void register_stage_3d_fp64(std::vector<StageEntry>& r);
void register_stage_3d_fp32(std::vector<StageEntry>& r);
void register_stage_visc_fp64(std::vector<StageEntry>& r);
void register_stage_visc_fp32(std::vector<StageEntry>& r);
void register_stage_char_fp64(std::vector<StageEntry>& r);

}  // namespace mfc
