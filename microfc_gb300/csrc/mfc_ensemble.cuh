// Ensemble of independent 2-D cases advanced together: one launch per RK
// stage over a work list of (case, tile) pairs, so 64 small cases of
// uneven size fill the GPU like one large one.  Each tile runs exactly the
// single-case tile code, so every case gets the same bits it would get
// alone.  The per-case parameter blocks travel in the kernel's parameter
// space (__grid_constant__), which keeps their fields in the constant bank.
#pragma once

#include <cuda_runtime.h>

#include <vector>

#include "mfc_device.cuh"
#include "mfc_pair.cuh"
#include "mfc_stage.cuh"

namespace mfc {

constexpr int kMaxEnsemble = 96;

struct EnsCase {
  DevParams P;
  double* reg[3];         // RK registers; reg[0] holds q_cons_ts(1)
  // split and gated: the primitive pairs (PrimPairs, mfc_pair.cuh) that the
  // first and the second stage of a step write and the next one reads; null:
  // there was no room for them
  f32x2* prim[2];
  double dt, dt_last;     // the case's dt and its (possibly trimmed) last-step dt
  int tiles_x, tile_base; // tiles per row, first tile in the work list
};

struct EnsParams {
  int num_cases, total_tiles, stage, time_stepper, last_step;
  // TMA maps of every case's stage inputs, [stage][case] (device memory; the
  // first stage's conservative register, then the pairs or, without them, the
  // other registers), for the tile variant launched; null: plain loads
  const TileMap* maps;
  // split WENO5: the coefficient record every cell of every case shares when
  // all cases have uniform grids (the FP32 records of a uniform grid do not
  // depend on its spacing); all off otherwise
  UniformCoefT<2> U;
  EnsCase c[kMaxEnsemble];
};
static_assert(sizeof(EnsParams) <= 32764, "ensemble parameters must fit the kernel parameter space");

// One block's tile of the work list.  One tile per block: the hardware deals
// the tiles out as blocks end, and the tile code keeps the registers that a
// persistent walk spent on its own state (it spilled 40 to 240 bytes).  24
// droplets of 128x64 to 512x256, us a step: persistent 387 (split) and 449
// (gated), with carried pairs 376 and 447, one tile per block 333 and 395.
// TMA: interior tiles arrive by one bulk tensor copy.
// VISC: every case carries its viscosity parameters (DevParams::visc).
// RT float: pair_tile with runs of RX and RY cells; double: stage_tile.
template <int NF, class RT, int TX, int TY, int NT, int RX, int RY, bool GATE, bool TMA, bool VISC>
__device__ __forceinline__ void ensemble_tile(const EnsParams& E) {
  static_assert(!TMA || sizeof(RT) == 4, "TMA loads are compiled for the split kernels");
  extern __shared__ __align__(128) unsigned char smem_raw[];
  const int t = blockIdx.x;
  int lo = 0, hi = E.num_cases - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (E.c[mid].tile_base <= t) lo = mid;
    else hi = mid - 1;
  }
  const EnsCase& C = E.c[lo];
  const int lt = t - C.tile_base;
  const int x0 = (lt % C.tiles_x) * TX, y0 = (lt / C.tiles_x) * TY;
  const double* in;
  double* out;
  int kind;
  if (E.stage == 0) {
    in = C.reg[0], out = C.reg[1], kind = kRkEuler;
  } else if (E.time_stepper == 2) {
    in = C.reg[1], out = C.reg[0], kind = kRk2Final;
  } else if (E.stage == 1) {
    in = C.reg[1], out = C.reg[2], kind = kRk3Mid;
  } else {
    in = C.reg[2], out = C.reg[0], kind = kRk3Final;
  }
  const TileMap* T = (TMA && E.maps != nullptr) ? E.maps + E.stage * E.num_cases + lo : nullptr;
  const double dt = E.last_step ? C.dt_last : C.dt;
  if constexpr (sizeof(RT) == 4) {
    const int64_t pitch = prim_pitch(C.P.n[0]);
    const PrimPairs B{E.stage == 0 ? nullptr : C.prim[E.stage - 1],
                      E.stage == E.time_stepper - 1 ? nullptr : C.prim[E.stage], pitch, pitch * C.P.n[1]};
    pair_tile<2, NF, TX, TY, NT, GATE, VISC, UniformCoefT<2>, TMA, RX, RY>(C.P, in, C.reg[0], out, dt, kind, x0, y0,
                                                                           smem_raw, &E.U, B, T, true);
  } else
    stage_tile<2, NF, 5, RT, TX, TY, NT, VISC>(C.P, in, C.reg[0], out, dt, kind, x0, y0, smem_raw);
}

template <int NF, class RT, int TX, int TY, int NT, int MINB, int RX, int RY, bool GATE, bool TMA, bool VISC>
__global__ void __launch_bounds__(NT, MINB) ensemble_stage_kernel(const __grid_constant__ EnsParams E) {
  ensemble_tile<NF, RT, TX, TY, NT, RX, RY, GATE, TMA, VISC>(E);
}

struct EnsembleEntry {
  int nf, wo, prec, tx, ty, nt;
  size_t smem, smem_shared_coef;  // dynamic shared memory: per-cell records / shared record
  const void* func;
  cudaError_t (*launch)(const EnsParams& E, int grid, size_t smem, cudaStream_t st);
  bool tma;    // interior tiles staged by TMA (needs EnsParams::maps)
  int box_w;   // x extent of the TMA box (cells), box_h rows
  int box_h;
  bool visc;   // compiled with the viscous terms
};

// MINB: blocks per SM that the registers must allow; RX, RY: run lengths of
// the split kernels.
template <int NF, class RT, int TX, int TY, int NT, int MINB, int RX = 1, int RY = 1, bool GATE = false,
          bool TMA = false, bool VISC = false>
EnsembleEntry ensemble_entry() {
  struct K {
    static constexpr auto func() { return &ensemble_stage_kernel<NF, RT, TX, TY, NT, MINB, RX, RY, GATE, TMA, VISC>; }
    static constexpr size_t smem(bool shared_coef) {
      if constexpr (sizeof(RT) == 4) return pair_smem<2, NF, TX, TY, NT, GATE, VISC, TMA>(shared_coef);
      else return stage_smem_total<2, NF, 5, RT, TX, TY, VISC, false>();
    }
  };
  EnsembleEntry e{};
  e.nf = NF;
  e.wo = 5;
  e.prec = sizeof(RT) == 8 ? 0 : (GATE ? 2 : 1);
  e.tx = TX;
  e.ty = TY;
  e.nt = NT;
  e.smem = K::smem(false);
  e.smem_shared_coef = K::smem(true);
  e.func = reinterpret_cast<const void*>(K::func());
  e.launch = [](const EnsParams& E, int grid, size_t smem, cudaStream_t st) {
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3((unsigned)grid);
    cfg.blockDim = dim3(NT);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, K::func(), E);
  };
  e.tma = TMA;
  e.box_w = TmaBox<TX, 3>::kWidth;
  e.box_h = TY + 6;
  e.visc = VISC;
  return e;
}

void register_ensemble_fp64(std::vector<EnsembleEntry>& r);
void register_ensemble_fp32(std::vector<EnsembleEntry>& r);
void register_ensemble_gated(std::vector<EnsembleEntry>& r);

}  // namespace mfc
