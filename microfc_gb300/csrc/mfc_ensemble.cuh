// Ensemble of independent 2-D cases advanced together: one persistent launch
// per RK stage walks a work list of (case, tile) pairs, so 64 small cases of
// uneven size fill the GPU like one large one.  Each tile runs exactly the
// single-case stage_tile, so every case gets the same bits it would get
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
  double dt, dt_last;     // the case's dt and its (possibly trimmed) last-step dt
  int tiles_x, tile_base; // tiles per row, first tile in the work list
};

struct EnsParams {
  int num_cases, total_tiles, stage, time_stepper, last_step;
  // TMA maps of every case's registers, [register][case] (device memory),
  // for the tile variant launched; null: plain loads
  const TileMap* maps;
  // split WENO5: the coefficient record every cell of every case shares when
  // all cases have uniform grids (the FP32 records of a uniform grid do not
  // depend on its spacing); all off otherwise
  UniformCoefT<2> U;
  EnsCase c[kMaxEnsemble];
};
static_assert(sizeof(EnsParams) <= 32764, "ensemble parameters must fit the kernel parameter space");

// One persistent block's walk over the work list (the body of both kernels).
// TMA: interior tiles arrive by one bulk tensor copy; the block initialises
// its mbarrier once and alternates its phase per copied tile.
// VISC: every case carries its viscosity parameters (DevParams::visc).
// RT float: pair_tile with runs of RX and RY cells; double: stage_tile.
template <int NF, class RT, int TX, int TY, int NT, int RX, int RY, bool GATE, bool TMA, bool VISC>
__device__ __forceinline__ void ensemble_walk(const EnsParams& E) {
  static_assert(!TMA || (sizeof(RT) == 4 && !VISC), "TMA loads are compiled for the inviscid split kernels");
  extern __shared__ __align__(128) unsigned char smem_raw[];
  uint32_t parity = 0;
  if constexpr (TMA) {
    if (E.maps != nullptr && threadIdx.x == 0)
      mbar_init(smem_addr(pair_staging<2, NF, TX, TY, VISC>(smem_raw) + PairShape<2, NF, TX, TY, VISC>::kStageBytes), 1);
    __syncthreads();
  }
  for (int t = blockIdx.x; t < E.total_tiles; t += gridDim.x) {
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
    int kind, reg;
    if (E.stage == 0) {
      in = C.reg[0], out = C.reg[1], kind = kRkEuler, reg = 0;
    } else if (E.time_stepper == 2) {
      in = C.reg[1], out = C.reg[0], kind = kRk2Final, reg = 1;
    } else if (E.stage == 1) {
      in = C.reg[1], out = C.reg[2], kind = kRk3Mid, reg = 1;
    } else {
      in = C.reg[2], out = C.reg[0], kind = kRk3Final, reg = 2;
    }
    const TileMap* T = (TMA && E.maps != nullptr) ? E.maps + reg * E.num_cases + lo : nullptr;
    const double dt = E.last_step ? C.dt_last : C.dt;
    if constexpr (sizeof(RT) == 4)
      pair_tile<2, NF, TX, TY, NT, GATE, VISC, UniformCoefT<2>, TMA, RX, RY>(
          C.P, in, C.reg[0], out, dt, kind, x0, y0, smem_raw, &E.U, PrimPairs{}, T, &parity);
    else
      stage_tile<2, NF, 5, RT, TX, TY, NT, VISC>(C.P, in, C.reg[0], out, dt, kind, x0, y0, smem_raw);
    __syncthreads();  // the next tile reuses the shared memory
  }
}

template <int NF, class RT, int TX, int TY, int NT, int MINB, int RX, int RY, bool GATE, bool TMA, bool VISC>
__global__ void __launch_bounds__(NT, MINB) ensemble_stage_kernel(const __grid_constant__ EnsParams E) {
  ensemble_walk<NF, RT, TX, TY, NT, RX, RY, GATE, TMA, VISC>(E);
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
    K::func()<<<grid, NT, smem, st>>>(E);
    return cudaGetLastError();
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
