// The split-precision RK stage with WENO5 (1-D and 2-D, with or without the
// learned gate and the viscous terms) on TX x TY tiles: what stage_tile does
// (mfc_stage.cuh), for variables kept in interleaved FP32 pairs.
//
// The FP32 units are far from busy here and so is HBM; a stage is bound by
// instruction issue and by what keeps the warps from it: barriers, the
// latency of shared memory and the special-function unit, and bursts of FP64
// (E - Pi, the RK sums).  Hence:
//
//   * both directions go through each phase together --
//     load + cons -> prim | (gate) | WENO x and y | HLLC x and y | divergence + RK
//     -- three barriers a tile instead of five, and phases of twice the items:
//     a 16x16 tile's reconstructions are exactly one run of nine for each of
//     256 threads;
//   * everything moves through shared memory as pairs (64-bit accesses), and
//     a reconstructing thread walks a run of cells: 13 loads for nine cells
//     instead of 45, one difference per cell instead of four;
//   * a face's fluxes and interface velocity overwrite the right values they
//     come from (no other face reads them), so both directions fit four
//     blocks per SM, whose threads may use 64 registers: no spills, where the
//     x-then-y order's five blocks of 48 had 44 bytes.
//
// The arithmetic of every value is that of the x-then-y order, so results do
// not depend on the tile shape.
//
// Measured (us a step; before: the x-then-y stage kernel with 16x16 tiles and
// TMA): split 100x50 22.8 -> 13.7, 333x167 32.3 -> 22.3, 1024x512 126 -> 110,
// 2048x1024 453 -> 403; gated 1024x512 145 -> 133, 2048x1024 504 -> 471;
// viscous split 1024x512 233 -> 194; 1-D 1000 cells 12.9 -> 9.6.  Counters at
// 2048x1024, first and later stages (121 and 140 us): issue 69 and 64 %, FP64
// unit 37 and 50 %, FMA 57 and 50 %, L1 45 and 42 %, DRAM 2.7 and 3.2 TB/s;
// per issue 2.2 to 2.3 warps wait at barriers, 1.7 for a fixed latency, 1.1 to
// 1.6 for shared memory, 1.2 for global loads.
#pragma once

#include "mfc_device.cuh"
#include "mfc_gate.cuh"
#include "mfc_stage.cuh"
#include "mfc_tma.cuh"

namespace mfc {

// Shared memory of the learned gate.  Its own region holds one flag per
// (cell, direction) reconstructed by the tile.  The gate phase's scratch --
// one 16x16 FP16 input block per warp, then the MLP's lane fragments
// (kGateFragWords words per lane, word-major) -- lives in the WENO value
// arrays, which are not written before the gate phase ends.
template <int ND, int TX, int TY, int NT>
struct GateShape {
  static constexpr int NGX = (TX + 2) * ((ND > 1) ? TY : 1);
  static constexpr int NGY = (ND > 1) ? TX * (TY + 2) : 0;
  static constexpr size_t kFragOff = size_t(NT / 32) * 512;
  static constexpr size_t kScratchBytes = kFragOff + size_t(kGateFragWords) * 32 * 4;
  static constexpr size_t kBytes = ((NGX + NGY + 15) / 16) * 16;
};

template <int ND, int NF, int TX, int TY, bool VISC>
struct PairShape {
  using Q = Eqs<ND, NF>;
  static constexpr int S = Q::S, H = 3, NPR = (S + 1) / 2;  // pairs; an odd last variable shares with a zero
  // (x runs read a column of rows at a time: the odd row length PCX of their
  // results keeps the stores free of bank conflicts; the primitive tile's rows
  // are as the copy engine lays them)
  static constexpr int TYE = ND > 1 ? TY : 1, LX = TX + 2 * H, LY = ND > 1 ? TY + 2 * H : 1;
  static constexpr int NCX = TX + 2, PCX = NCX | 1, NCY = ND > 1 ? TY + 2 : 0;
  // sizes in pairs: primitive tile, left and right values of each direction
  static constexpr int NQ = NPR * LY * LX, NWX = NPR * TYE * PCX, NWY = NPR * NCY * TX;
  static constexpr int align16(int n) { return (n + 1) / 2 * 2; }
  static constexpr int OWX = align16(NQ), OWY = OWX + 2 * NWX, OEND = align16(OWY + 2 * NWY);
  // rows of a face's result: the fluxes, the interface velocity and the
  // viscous x-momentum, y-momentum and energy; pair k sits in right-value
  // slot k, beyond NPR in left-value slot k - NPR
  static constexpr int NR = S + 1 + (VISC ? 3 : 0), NRP = (NR + 1) / 2;
  static_assert(NRP <= 2 * NPR, "a face's results must fit its two states");
  static constexpr size_t kMainBytes = sizeof(f32x2) * size_t(OEND);
  static constexpr size_t kCoefBytes = sizeof(float) * size_t(kCoefRec) * (NCX + NCY);
  // TMA staging: the FP64 box of all variables in the value arrays
  static constexpr uint32_t kStageBytes = uint32_t(TmaBox<TX, H>::kWidth) * LY * S * 8;
};

// Offset of the gate's flags and, after them, of the per-cell coefficient
// records: past a TMA kernel's staging area, which is filled while they are.
template <int ND, int NF, int TX, int TY, bool VISC, bool TMA>
constexpr size_t pair_gate_offset() {
  using Sh = PairShape<ND, NF, TX, TY, VISC>;
  constexpr size_t t = (sizeof(f32x2) * size_t(Sh::OWX) + 128 + Sh::kStageBytes + 16 + 15) / 16 * 16;
  return TMA && t > Sh::kMainBytes ? t : Sh::kMainBytes;
}
template <int ND, int NF, int TX, int TY, int NT, bool GATE, bool VISC, bool TMA>
constexpr size_t pair_coef_offset() {
  return pair_gate_offset<ND, NF, TX, TY, VISC, TMA>() + (GATE ? GateShape<ND, TX, TY, NT>::kBytes : 0);
}
// Dynamic shared memory of one block (without the records on a uniform grid).
template <int ND, int NF, int TX, int TY, int NT, bool GATE, bool VISC, bool TMA>
constexpr size_t pair_smem(bool shared_coef) {
  return pair_coef_offset<ND, NF, TX, TY, NT, GATE, VISC, TMA>() +
         (shared_coef ? 0 : PairShape<ND, NF, TX, TY, VISC>::kCoefBytes);
}
// The TMA staging area: after the primitive tile, 128-byte aligned, the box,
// then its mbarrier and a flag.
template <int ND, int NF, int TX, int TY, bool VISC>
__device__ __forceinline__ unsigned char* pair_staging(unsigned char* smem_raw) {
  using Sh = PairShape<ND, NF, TX, TY, VISC>;
  const uintptr_t a = reinterpret_cast<uintptr_t>(smem_raw + Sh::OWX * sizeof(f32x2));
  return reinterpret_cast<unsigned char*>((a + 127) & ~uintptr_t(127));
}

// The primitive pairs of a 2-D state in global memory: pair k of cell (x, y)
// at (k * rows + y) * pitch + x + 1 (one column of lead, so that a tile's
// 22-cell rows, which start at x0 - 3, start on 16 bytes).  A stage that is
// given `out` converts the state it makes, in registers, and writes the pairs;
// the next stage, given them as `in`, loads FP32 pairs in place of FP64
// conservative values: half the bytes of a tile, no conversion of its halo
// (448 cells for 256), and interior tiles arrive in their final layout by one
// bulk copy.  The conversion is the same, so the bits are too.
// 3-D (mfc_pair_sweep.cuh): pair k of cell o at k * sv + o; cur: in, or where
// the x sweep puts the pairs of a state that comes without.
struct PrimPairs {
  const f32x2* in;
  f32x2* out;
  int64_t pitch, plane;
  f32x2* cur;
};
__host__ __device__ inline int64_t prim_pitch(int nx) { return (nx + 2 + 15) / 16 * 16; }

// One tile of one RK stage; the tile's first cell is (x0, y0).  U: shared
// coefficient records; T: the TMA map of B.in, or of the stage input where
// that is null (TMA kernels), in the kernel's parameters or, map_in_memory
// (the ensemble's), in global memory.
template <int ND, int NF, int TX, int TY, int NT, bool GATE, bool VISC, class UC, bool TMA, int RX, int RY>
__device__ __forceinline__ void pair_tile(const DevParams& P, const double* __restrict__ qin,
                                          const double* __restrict__ qbase, double* __restrict__ qout,
                                          const double dt, const int kind, const int x0, const int y0,
                                          unsigned char* smem_raw, const UC* U, const PrimPairs& B,
                                          const TileMap* T = nullptr, const bool map_in_memory = false) {
  using Sh = PairShape<ND, NF, TX, TY, VISC>;
  using Q = Eqs<ND, NF>;
  constexpr int S = Sh::S, H = Sh::H, NPR = Sh::NPR, LX = Sh::LX, LY = Sh::LY, TYE = Sh::TYE;
  constexpr int NCX = Sh::NCX, PCX = Sh::PCX, NCY = Sh::NCY, NRP = Sh::NRP, HY = ND > 1 ? H : 0;
  constexpr int WX = TX + 2 * H;  // cells of a tile row (LX: its length in shared memory)
  constexpr int CPT = (TX * TYE + NT - 1) / NT;  // cells per thread in the last phase

  f32x2* const sq = reinterpret_cast<f32x2*>(smem_raw);  // [pair][LY][LX]
  f32x2* const wxl = sq + Sh::OWX;                        // [pair][TYE][NCX]
  f32x2* const wxr = wxl + Sh::NWX;
  f32x2* const wyl = sq + Sh::OWY;                        // [pair][NCY][TX]
  f32x2* const wyr = wyl + Sh::NWY;
  float* const scx =
      reinterpret_cast<float*>(smem_raw + pair_coef_offset<ND, NF, TX, TY, NT, GATE, VISC, TMA>());
  float* const scy = scx + kCoefRec * NCX;
  auto qi = [](int pr, int ly, int lx) { return (pr * LY + ly) * LX + lx; };
  auto wxi = [](int pr, int ty, int cx) { return (pr * TYE + ty) * PCX + cx; };
  auto wyi = [](int pr, int cy, int tx) { return (pr * NCY + cy) * TX + tx; };
  // pair k of the results of x face f (left of cell f) and of y face f
  auto fx = [&](int k, int ty, int f) -> f32x2& {
    return k < NPR ? wxr[wxi(k, ty, f)] : wxl[wxi(k - NPR, ty, f + 1)];
  };
  auto fy = [&](int k, int f, int tx) -> f32x2& {
    return k < NPR ? wyr[wyi(k, f, tx)] : wyl[wyi(k - NPR, f + 1, tx)];
  };
  (void)fy;
  (void)wyi;
  // variable v of the primitive tile
  auto prim = [&](int v, int ly, int lx) { return reinterpret_cast<const float*>(sq)[qi(v >> 1, ly, lx) * 2 + (v & 1)]; };

  const int tid = threadIdx.x;
  const int nx = P.n[0], ny = P.n[1];
  const double one = fma64_unit(P.inv_d[0]).one;  // the FP64 sums' register operand
  float gam_i[NF], pi_i[NF];
#pragma unroll
  for (int f = 0; f < NF; ++f) {
    gam_i[f] = P.gammas_f[f];
    pi_i[f] = P.pi_infs_f[f];
  }
  // a uniform grid: every cell of a direction shares one coefficient record,
  // read from the kernel parameters
  const bool uni = U->on[0] != 0 && (ND < 2 || U->on[ND > 1 ? 1 : 0] != 0);

  // ---- load + BCs + cons -> prim ------------------------------------------------
  // the per-cell records come from constant tables: before the wait
  for (int it = uni ? kCoefRec * NCX : tid; it < kCoefRec * NCX; it += NT) {
    const int cx = it % NCX, k = it / NCX;
    scx[cx * kCoefRec + k] =
        k < kNumCoef ? d2f_bits(__ldg(P.coef[0] + k * P.cstride[0] + clamp_coef_index(x0 - 1 + cx, nx) + P.coff)) : 0.f;
  }
  if constexpr (ND > 1) {
    for (int it = uni ? kCoefRec * NCY : tid; it < kCoefRec * NCY; it += NT) {
      const int cy = it % NCY, k = it / NCY;
      scy[cy * kCoefRec + k] =
          k < kNumCoef ? d2f_bits(__ldg(P.coef[1] + k * P.cstride[1] + clamp_coef_index(y0 - 1 + cy, ny) + P.coff))
                       : 0.f;
    }
  }
  // one cell of the tile: BCs already applied, cons -> prim into the tile
  auto store_prim = [&](const double (&q)[S], const int ly, const int lx) {
    float pr[S];
    cons_to_prim_split<ND, NF>(q, P, one, pr);
#pragma unroll
    for (int k = 0; k < NPR; ++k) sq[qi(k, ly, lx)] = f2_pack(pr[2 * k], 2 * k + 1 < S ? pr[2 * k + 1 < S ? 2 * k + 1 : 0] : 0.f);
  };
  // corners are never read, except the four diagonal neighbours of the tile
  // that the viscous cross derivatives use
  auto unused_corner = [](const int lx, const int ly) {
    const bool hx = lx < H || lx >= H + TX;
    const bool hy = ND > 1 && (ly < H || ly >= H + TY);
    return hx && hy && !(VISC && (lx == H - 1 || lx == H + TX) && (ly == H - 1 || ly == H + TY));
  };

  // TMA staging: a tile whose halo lies inside the domain (no boundary
  // condition, no processor halo) arrives in one bulk tensor copy of all
  // variables into the value arrays, which are free until the WENO phase.
  bool use_tma = false;
  unsigned char* stg = nullptr;
  uint32_t bar = 0;
  using Box = TmaBox<TX, H>;
  if constexpr (TMA) {
    static_assert(ND == 2, "TMA loads are compiled for the 2-D kernel");
    use_tma = T != nullptr && T->on && x0 >= H && x0 + TX + H <= nx && y0 >= H && y0 + TY + H <= ny;
    if (use_tma) {
      stg = pair_staging<ND, NF, TX, TY, VISC>(smem_raw);  // B.in: only its barrier and flag are used
      bar = smem_addr(stg + Sh::kStageBytes);
      if (tid == 0) mbar_init(bar, 1);
    }
  }
  griddep_wait();  // the state below is the previous stage's output
  if (kind != kRkEuler && kind != kRhsOnly) {
    // the RK base register's rows of the tile, read only by the last phase:
    // every 128-byte line prefetched into L2 while the tile is worked on
    constexpr int kLines = (TX * 8 + 127) / 128;
    for (int it = tid; it < S * TYE * kLines; it += NT) {
      const int line = it % kLines, r = it / kLines, ty = r % TYE, v = r / TYE;
      const int gx = x0 + line * 16, gy = ND > 1 ? y0 + ty : 0;
      if (gx >= nx || gy >= ny) continue;
      asm volatile("prefetch.global.L2 [%0];" ::"l"(qbase + gy * P.sy + gx + v * P.sv));
    }
  }
  // The learned gate's flags, one per (cell, direction).  The first stage of a
  // time step (and an RHS evaluation) runs the network below; with
  // P.gate_flags it also stores the decisions, and the step's later stages
  // read them back here, while the tile is on its way: the gate judges each
  // cell once per time step, on the state at t^n.  Every stored position
  // (including the ghost positions x = -1, nx and y = -1, ny next to the
  // domain) is written by exactly one tile.
  constexpr int NG = GateShape<ND, TX, TY, NT>::NGX + GateShape<ND, TX, TY, NT>::NGY;
  uint8_t* const gflag = smem_raw + pair_gate_offset<ND, NF, TX, TY, VISC, TMA>();
  const bool stored_flags = GATE && P.gate_flags != nullptr && kind != kRkEuler && kind != kRhsOnly;
  // position p of the tile: its slot in the stored planes (false: beyond the
  // planes, a cell of a partial edge tile whose results are not kept) and
  // whether this tile is the one that stores it
  auto flag_slot = [&](const int p, int64_t& slot, bool& owner) {
    constexpr int NGX = GateShape<ND, TX, TY, NT>::NGX;
    if (p < NGX) {
      const int cx = p % NCX, ty = p / NCX;
      const int gx = x0 - 1 + cx, gy = y0 + ty;
      slot = (int64_t)gy * (nx + 2) + (gx + 1);
      owner = (cx >= 1 && cx <= TX) || gx == -1 || gx == nx;
      return gx >= -1 && gx <= nx && gy < ny;
    }
    const int p2 = p - NGX, tx = p2 % TX, cy = p2 / TX;
    const int gx = x0 + tx, gy = y0 - 1 + cy;
    slot = (int64_t)ny * (nx + 2) + (int64_t)(gy + 1) * nx + gx;
    owner = (cy >= 1 && cy <= TY) || gy == -1 || gy == ny;
    return gx < nx && gy >= -1 && gy <= ny;
  };
  if (stored_flags) {
    for (int p = tid; p < NG; p += NT) {
      int64_t slot;
      bool owner;
      gflag[p] = flag_slot(p, slot, owner) ? __ldg(P.gate_flags + slot) : uint8_t(1);
    }
  }
  if (use_tma) {
    volatile int* landed = reinterpret_cast<volatile int*>(stg + Sh::kStageBytes + 8);
    if (tid == 0) {
      if (map_in_memory) tensormap_acquire(&T->map);
      if (B.in != nullptr) {
        mbar_arrive_expect_tx(bar, uint32_t(Sh::NQ * sizeof(f32x2)));
        tma_load_3d(smem_addr(sq), &T->map, x0 - H + 1, y0 - H, 0, bar);
      } else {
        mbar_arrive_expect_tx(bar, Sh::kStageBytes);
        tma_load_3d(smem_addr(stg), &T->map, x0 - Box::kLead, y0 - H, 0, bar);
      }
      const bool ok = mbar_wait_bounded(bar, 0, 1000000000ull);  // 1 s
      if (!ok) (void)mbar_wait_bounded(bar, 0, 1000000000ull);    // the copy may still be in flight
      *landed = ok ? 1 : 0;
    }
    __syncthreads();
    if (*landed == 0) {
      if (tid == 0 && P.status) atomicOr(P.status, MFC_FLAG_TIMEOUT);
      return;
    }
    (void)mbar_try_wait(bar, 0);  // completed: each thread acquires the copy's writes
    const double* sd = reinterpret_cast<const double*>(stg);
    for (int c = B.in != nullptr ? WX * LY : tid; c < WX * LY; c += NT) {
      const int lx = c % WX, ly = c / WX;
      if (unused_corner(lx, ly)) continue;
      double q[S];
#pragma unroll
      for (int v = 0; v < S; ++v) q[v] = sd[(v * LY + ly) * Box::kWidth + lx + (Box::kLead - H)];
      store_prim(q, ly, lx);
    }
  } else if (ND == 2 && B.in != nullptr) {
    // the stored pairs, with the boundary conditions (a reflected cell's
    // normal velocity negated: the conversion is odd in the momentum)
    for (int c = tid; c < WX * LY; c += NT) {
      const int lx = c % WX, ly = c / WX;
      if (unused_corner(lx, ly)) continue;
      bool flip_x = false, flip_y = false;
      const int gx = map_cell(x0 - H + lx, nx, P.bc_beg[0], P.bc_end[0], &flip_x);
      const int gy = map_cell(y0 - H + ly, ny, P.bc_beg[1], P.bc_end[1], &flip_y);
      const f32x2* src = B.in + gy * B.pitch + gx + 1;
#pragma unroll
      for (int k = 0; k < NPR; ++k) {
        f32x2 w = __ldg(src + k * B.plane);
        constexpr f32x2 lo = 0x80000000ull, hi = lo << 32;
        if (k == Q::MOM / 2 && flip_x) w ^= Q::MOM % 2 ? hi : lo;
        if (k == (Q::MOM + 1) / 2 && flip_y) w ^= (Q::MOM + 1) % 2 ? hi : lo;
        sq[qi(k, ly, lx)] = w;
      }
    }
  } else {  // plain loads, with the boundary conditions and processor halos
    for (int c = tid; c < WX * LY; c += NT) {
      const int lx = c % WX, ly = c / WX;
      if (unused_corner(lx, ly)) continue;
      bool flip_x, flip_y;
      int64_t vs;
      const double* src = tile_cell<ND, H>(P, qin, x0 - H + lx, ND > 1 ? y0 - H + ly : 0, vs, flip_x, flip_y);
      double q[S];
#pragma unroll
      for (int v = 0; v < S; ++v) q[v] = __ldg(src + v * vs);
      if (flip_x) q[Q::MOM] = -q[Q::MOM];
      if (ND > 1 && flip_y) q[Q::MOM + 1] = -q[Q::MOM + 1];
      store_prim(q, ly, lx);
    }
  }
  __syncthreads();

  // ---- learned gate: the network on every reconstructed position of the tile ------
  if constexpr (GATE) {
    if (!stored_flags) {
      using G = GateShape<ND, TX, TY, NT>;
      static_assert(G::kScratchBytes <= sizeof(f32x2) * size_t(Sh::OEND - Sh::OWX),
                    "the gate's scratch must fit the value arrays");
      unsigned char* scratch = reinterpret_cast<unsigned char*>(wxl);
      __half* gin = reinterpret_cast<__half*>(scratch);
      uint32_t* frag = reinterpret_cast<uint32_t*>(scratch + G::kFragOff);
      const int warp = tid >> 5, lane = tid & 31;
      const uint32_t* gsrc =
          reinterpret_cast<const uint32_t*>(static_cast<const unsigned char*>(P.gate_w) + kGateFragOffset);
      for (int i = tid; i < kGateFragWords * 8; i += NT)
        reinterpret_cast<uint4*>(frag)[i] = __ldg(reinterpret_cast<const uint4*>(gsrc) + i);
      __syncthreads();
      const GateFragsSmem F{frag + 4 * lane};
      __half* my = gin + warp * 256;
      constexpr int NCH = (NG + 15) / 16;
      for (int ch = warp; ch < NCH; ch += NT / 32) {
        const int cell = ch * 16 + (lane & 15);
        const int var = lane < 16 ? Q::ADV : Q::E;  // alpha_1 | pressure
        float s[5] = {0.f, 0.f, 0.f, 0.f, 0.f};
        if (cell < G::NGX) {
          const int cx = cell % NCX, ty = cell / NCX;
#pragma unroll
          for (int k = 0; k < 5; ++k) s[k] = prim(var, ty + HY, cx + H - 1 + k - 2);
        } else if (cell < NG) {
          const int c2 = cell - G::NGX, tx = c2 % TX, cy = c2 / TX;
#pragma unroll
          for (int k = 0; k < 5; ++k) s[k] = prim(var, cy + H - 1 + k - 2, tx + H);
        }
        float xf[5];
        gate_norm5_var(s, xf, lane < 16 ? 0 : 1);
        // columns 0..7 (alpha_1) or 8..15 (pressure) of the cell's row: five
        // features and three zeros, one 16-byte store
        const uint4 half8 = make_uint4(pack_h2(xf[0], xf[1]), pack_h2(xf[2], xf[3]), pack_h2(xf[4], 0.f), 0u);
        reinterpret_cast<uint4*>(my + (lane & 15) * 16)[lane >> 4] = half8;
        __syncwarp();
        float lo, hi;
        gate_mlp16(my, F, lo, hi);
        if ((lane & 3) == 0) {
          const int c_lo = ch * 16 + (lane >> 2), c_hi = c_lo + 8;
          if (c_lo < NG) gflag[c_lo] = lo > 0.f;
          if (c_hi < NG) gflag[c_hi] = hi > 0.f;
        }
        __syncwarp();
      }
      __syncthreads();
      if (P.gate_flags != nullptr && kind == kRkEuler) {
        // the first stage stores the decisions of the positions it owns
        for (int p = tid; p < NG; p += NT) {
          int64_t slot;
          bool owner;
          if (flag_slot(p, slot, owner) && owner) P.gate_flags[slot] = gflag[p];
        }
      }
    }
  }

  // ---- WENO: cells x0-1 .. x0+TX of the rows, y0-1 .. y0+TY of the columns ----
  // A thread takes a run of RX (RY) consecutive cells of one row (column) and
  // one pair of variables: each value is loaded once and each difference
  // formed once, instead of five and four times.
  {
    static_assert(NCX % RX == 0 && (ND < 2 || NCY % RY == 0), "runs must fill the rows and columns");
    constexpr int NXR = TYE * (NCX / RX), NYR = ND > 1 ? TX * (NCY / RY) : 0;  // runs per pair
    const f32x2 eps2 = f2_pack(P.weno_eps_f, P.weno_eps_f);
    // coef(j, use): calls use(C) with C(k) = coefficient k of the run's cell j
    // as a (c, c) pair; gate(j): whether cell j takes the nonlinear weights
    auto run = [&](auto len, const f32x2* at, const int st, f32x2* l, f32x2* r, const int ost, auto&& coef,
                   auto&& gate) {
      f32x2 v1 = at[-st], v2 = at[0], v3 = at[st];
      f32x2 dm2 = f2_sub(v1, at[-2 * st]), dm1 = f2_sub(v2, v1), d0 = f2_sub(v3, v2);
      constexpr int kUnroll = GATE ? 1 : 3;  // code size: fully unrolled is no faster, and slower with both branches
#pragma unroll kUnroll
      for (int j = 0; j < decltype(len)::value; ++j) {
        const f32x2 v4 = at[(j + 2) * st], d1 = f2_sub(v4, v3);
        f32x2 vl, vr;
        coef(j, [&](const auto& C) {
          if constexpr (GATE) {
            if (gate(j)) weno5_pair_diffs(C, v2, d1, d0, dm1, dm2, eps2, vl, vr);
            else weno5_pair_linear(C, v2, d1, d0, dm1, dm2, vl, vr);
          } else {
            weno5_pair_diffs(C, v2, d1, d0, dm1, dm2, eps2, vl, vr);
          }
        });
        l[j * ost] = vl;
        r[j * ost] = vr;
        v2 = v3;
        v3 = v4;
        dm2 = dm1;
        dm1 = d0;
        d0 = d1;
      }
    };
    // UNI: the shared records, else the cell's staged record
    auto runs = [&](auto uni) {
      constexpr bool UNI = decltype(uni)::value;
      auto record = [](const float* rec, auto&& use) {
        float c[kCoefRec];
        load_coef_record(rec, c);
        use([&](int k) { return f2_pack(c[k], c[k]); });
      };
      for (int it = tid; it < NPR * (NXR + NYR); it += NT) {
        if (it < NPR * NXR) {
          const int ty = it % TYE, q = it / TYE, w = q % NPR, c0 = q / NPR * RX;
          run(KindC<RX>{}, sq + qi(w, ty + HY, c0 + H - 1), 1, wxl + wxi(w, ty, c0), wxr + wxi(w, ty, c0), 1,
              [&](int j, auto&& use) {
                if constexpr (UNI) use([&](int k) { return f32x2(U->rec[0][k]); });
                else record(scx + (c0 + j) * kCoefRec, use);
              },
              [&](int j) { return gflag[ty * NCX + c0 + j] != 0; });
        } else if constexpr (ND > 1) {
          const int i2 = it - NPR * NXR, tx = i2 % TX, q = i2 / TX, w = q % NPR, c0 = q / NPR * RY;
          run(KindC<RY>{}, sq + qi(w, c0 + H - 1, tx + H), LX, wyl + wyi(w, c0, tx), wyr + wyi(w, c0, tx), TX,
              [&](int j, auto&& use) {
                if constexpr (UNI) use([&](int k) { return f32x2(U->rec[ND > 1 ? 1 : 0][k]); });
                else record(scy + (c0 + j) * kCoefRec, use);
              },
              [&](int j) { return gflag[TYE * NCX + (c0 + j) * TX + tx] != 0; });
        }
      }
    };
    if (uni) runs(FlagC<true>{});
    else runs(FlagC<false>{});
  }
  __syncthreads();

  // ---- HLLC: x faces x0-1/2 .. x0+TX-1/2, then y faces -------------------------------
  {
    constexpr int NFX = TYE * (TX + 1), NFY = ND > 1 ? (TY + 1) * TX : 0;
    auto states = [&](const f32x2* r, const f32x2* l, const int step, const bool lfr, const bool rfl, float (&qL)[S],
                      float (&qR)[S]) {
#pragma unroll
      for (int k = 0; k < NPR; ++k) {
        float a0, a1, b0, b1;
        f2_unpack(r[k * step], a0, a1);
        f2_unpack(l[k * step], b0, b1);
        qL[2 * k] = a0;
        qR[2 * k] = b0;
        if (2 * k + 1 < S) {
          qL[2 * k + 1 < S ? 2 * k + 1 : 0] = a1;
          qR[2 * k + 1 < S ? 2 * k + 1 : 0] = b1;
        }
      }
      if (lfr || rfl) {  // Riemann-state extrapolation at a domain face (bc -4)
#pragma unroll
        for (int v = 0; v < S; ++v) {
          const float a = qL[v], b = qR[v];
          qL[v] = lfr ? b : a;
          qR[v] = rfl ? a : b;
        }
      }
    };
    // the results of a face: R[0 .. NR-1]
    auto pair_of = [](const float (&R)[2 * NRP], const int k) { return f2_pack(R[2 * k], R[2 * k + 1]); };
    auto U_ = [&](int c, int x, int y) { return prim(Q::MOM + c, y, x); };
    for (int it = tid; it < NFX + NFY; it += NT) {
      float qL[S], qR[S], F[S], us, R[2 * NRP];
      R[2 * NRP - 1] = 0.f;
      if (it < NFX) {
        const int f = it % (TX + 1), ty = it / (TX + 1);
        const int gface = x0 - 1 + f;  // face gface+1/2
        states(wxr + wxi(0, ty, f), wxl + wxi(0, ty, f + 1), TYE * PCX, gface == -1 && P.bc_beg[0] == -4,
               gface == nx - 1 && P.bc_end[0] == -4, qL, qR);
        if constexpr (VISC) {
          float vs[ND], dxv[2] = {0.f, 0.f}, dyv[2] = {0.f, 0.f}, vf[3];
          hllc_face<ND, NF, 0, float, true>(qL, qR, gam_i, pi_i, F, us, vs);
          const ViscParams& V = *P.visc;
          if (V.fg[0] != nullptr) {
            // weno_Re_flux = T: the prepared face gradients (clamped indices
            // for the rows and faces of partial tiles, whose results are dropped)
            const int gy = ND > 1 ? min(y0 + ty, ny - 1) : 0;
            const int64_t plane = (int64_t)(ND > 1 ? ny : 1) * (nx + 1);
            const int64_t o = (int64_t)gy * (nx + 1) + (min(max(gface, -1), nx - 1) + 1);
            if constexpr (ND > 1) {  // pairs of the two components
              const f32x2* g = reinterpret_cast<const f32x2*>(V.fg[0]) + o;
              f2_unpack(__ldg(g), dxv[0], dxv[1]);
              f2_unpack(__ldg(g + plane), dyv[0], dyv[1]);
            } else {
              dxv[0] = d2f_bits(__ldg(V.fg[0] + o));
            }
          } else {
            const int ly = ty + HY, lx = f + H - 1;  // the face's left cell
            const auto Dx = divisor(d2f_bits(__ldg(V.dcc[0] + min(x0 + f, nx))));  // x_cc(j+1) - x_cc(j)
#pragma unroll
            for (int c = 0; c < ND; ++c) {
              const float g = div_rn(U_(c, lx + 1, ly) - U_(c, lx, ly), Dx);
              dxv[c] = 0.5f * (g + g);
            }
            if constexpr (ND > 1) {
              const int gy = min(y0 + ty, ny - 1);
              const auto D0 = divisor(d2f_bits(__ldg(V.dcc[1] + gy))), D1 = divisor(d2f_bits(__ldg(V.dcc[1] + gy + 1)));
#pragma unroll
              for (int c = 0; c < ND; ++c) {
                auto Ly = [&](int x) { return div_rn(U_(c, x, ly) - U_(c, x, ly - 1), D0); };
                auto Ry = [&](int x) { return div_rn(U_(c, x, ly + 1) - U_(c, x, ly), D1); };
                const float A = 0.25f * (Ly(lx + 1) + Ry(lx + 1) + Ly(lx) + Ry(lx));
                dyv[c] = 0.5f * (A + A);
              }
            }
          }
          viscous_face_flux<ND, NF, 0, float>(qL, qR, V, vs, dxv, dyv, vf);
#pragma unroll
          for (int t = 0; t < 3; ++t) R[S + 1 + t] = vf[t];
        } else {
          hllc_face_fast<ND, NF, 0>(qL, qR, gam_i, pi_i, F, us);
        }
#pragma unroll
        for (int v = 0; v < S; ++v) R[v] = F[v];
        R[S] = us;
#pragma unroll
        for (int k = 0; k < NRP; ++k) fx(k, ty, f) = pair_of(R, k);
      } else if constexpr (ND > 1) {
        const int i2 = it - NFX, tx = i2 % TX, f = i2 / TX;
        const int gface = y0 - 1 + f;
        states(wyr + wyi(0, f, tx), wyl + wyi(0, f + 1, tx), NCY * TX, gface == -1 && P.bc_beg[1] == -4,
               gface == ny - 1 && P.bc_end[1] == -4, qL, qR);
        if constexpr (VISC) {
          float vs[ND], dxv[2], dyv[2], vf[3];
          hllc_face<ND, NF, 1, float, true>(qL, qR, gam_i, pi_i, F, us, vs);
          const ViscParams& V = *P.visc;
          const int gx = min(x0 + tx, nx - 1);
          if (V.fg[1] != nullptr) {
            // weno_Re_flux = T: the prepared face gradients
            const f32x2* g = reinterpret_cast<const f32x2*>(V.fg[1]) +
                             (int64_t)(min(max(gface, -1), ny - 1) + 1) * nx + gx;
            f2_unpack(__ldg(g), dxv[0], dxv[1]);
            f2_unpack(__ldg(g + (int64_t)(ny + 1) * nx), dyv[0], dyv[1]);
          } else {
            const int ly = f + H - 1, lx = tx + H;  // the face's lower cell
            const auto Dy = divisor(d2f_bits(__ldg(V.dcc[1] + min(y0 + f, ny))));  // y_cc(k+1) - y_cc(k)
            const auto D0 = divisor(d2f_bits(__ldg(V.dcc[0] + gx))), D1 = divisor(d2f_bits(__ldg(V.dcc[0] + gx + 1)));
#pragma unroll
            for (int c = 0; c < 2; ++c) {
              auto Lx = [&](int y) { return div_rn(U_(c, lx, y) - U_(c, lx - 1, y), D0); };
              auto Rx = [&](int y) { return div_rn(U_(c, lx + 1, y) - U_(c, lx, y), D1); };
              const float A = 0.25f * (Lx(ly + 1) + Rx(ly + 1) + Lx(ly) + Rx(ly));
              dxv[c] = 0.5f * (A + A);
              const float g = div_rn(U_(c, lx, ly + 1) - U_(c, lx, ly), Dy);
              dyv[c] = 0.5f * (g + g);
            }
          }
          viscous_face_flux<ND, NF, 1, float>(qL, qR, V, vs, dxv, dyv, vf);
#pragma unroll
          for (int t = 0; t < 3; ++t) R[S + 1 + t] = vf[t];
        } else {
          hllc_face_fast<ND, NF, 1>(qL, qR, gam_i, pi_i, F, us);
        }
#pragma unroll
        for (int v = 0; v < S; ++v) R[v] = F[v];
        R[S] = us;
#pragma unroll
        for (int k = 0; k < NRP; ++k) fy(k, f, tx) = pair_of(R, k);
      }
    }
  }
  __syncthreads();

  // ---- flux divergence, RK combination, store ------------------------------------------
  griddep_launch_dependents();
  bool bad = false;
  const float dtf = __double2float_rn(dt);  // the increments are FP32
  double icfl = 0.0;
  // KIND: the stage's combination as a compile-time constant, chosen once
  // per block rather than once per cell and variable
  auto finish = [&](auto kind_c) {
    constexpr int KIND = decltype(kind_c)::value;
#pragma unroll
    for (int k = 0; k < CPT; ++k) {
      const int e = tid + k * NT;
      if (e >= TX * TYE) break;
      const int tx = e % TX, ty = e / TX;
      const int gx = x0 + tx, gy = y0 + ty;
      if (gx >= nx || (ND > 1 && gy >= ny)) continue;
      const int64_t o = gy * P.sy + gx;
      double base[S], in[S];  // all loads in flight before the divergence
      if constexpr (KIND != kRhsOnly) {
#pragma unroll
        for (int v = 0; v < S; ++v) base[v] = __ldg(qbase + o + v * P.sv);
        if constexpr (KIND != kRkEuler) {
#pragma unroll
          for (int v = 0; v < S; ++v) in[v] = __ldg(qin + o + v * P.sv);
        }
      }
      float rhs[S], d[2 * NRP], du;
      // F(face0) - F(face1) of every row, and the velocity difference the other way
      auto diff = [&](auto&& face0, auto&& face1) {
#pragma unroll
        for (int r = 0; r < NRP; ++r) {
          const f32x2 a = face0(r), b = face1(r);
          f2_unpack(f2_sub(a, b), d[2 * r], d[2 * r + 1]);
          if (r == S / 2) {
            float a0, a1, b0, b1;
            f2_unpack(a, a0, a1);
            f2_unpack(b, b0, b1);
            du = S % 2 ? b1 - a1 : b0 - a0;
          }
        }
      };
      // the source term of volume fraction f and the viscous rows
      // (m_rhs.fpp:591-603, 639-651) of one direction
      auto sources = [&](const float inv) {
#pragma unroll
        for (int f = 0; f < NF; ++f) {
          const float a = prim(Q::ADV + f, ty + HY, tx + H);
          rhs[Q::ADV + f] = mul_add(inv * a, du, rhs[Q::ADV + f]);
        }
        if constexpr (VISC) {
#pragma unroll
          for (int t = 0; t <= ND; ++t) {
            const int v = t < ND ? Q::MOM + t : Q::E, r = S + 1 + (t < ND ? t : 2);
            rhs[v] = mul_add(inv, d[r], rhs[v]);
          }
        }
      };
      const float ix = d2f_ftz(__ldg(P.inv_d[0] + gx));
      diff([&](int r) { return fx(r, ty, tx); }, [&](int r) { return fx(r, ty, tx + 1); });
#pragma unroll
      for (int v = 0; v < S; ++v) rhs[v] = ix * d[v];
      sources(ix);
      if constexpr (ND > 1) {
        const float iy = d2f_ftz(__ldg(P.inv_d[1] + gy));
        diff([&](int r) { return fy(r, ty, tx); }, [&](int r) { return fy(r, ty + 1, tx); });
#pragma unroll
        for (int v = 0; v < S; ++v) rhs[v] = mul_add(iy, d[v], rhs[v]);
        sources(iy);
      }
      double out[S];
#pragma unroll
      for (int v = 0; v < S; ++v) {
        if constexpr (KIND == kRhsOnly) out[v] = f2d_bits(rhs[v]);
        else out[v] = rk_combine_split(KIND, base[v], KIND == kRkEuler ? base[v] : in[v], dtf, rhs[v], one);
        bad |= not_finite(out[v]);
        qout[o + v * P.sv] = out[v];
      }
      if (ND == 2 && KIND != kRhsOnly && B.out != nullptr) {
        float pr[S];
        cons_to_prim_split<ND, NF>(out, P, one, pr);
        f32x2* dst = B.out + gy * B.pitch + gx + 1;
#pragma unroll
        for (int k = 0; k < NPR; ++k)
          dst[k * B.plane] = f2_pack(pr[2 * k], 2 * k + 1 < S ? pr[2 * k + 1 < S ? 2 * k + 1 : 0] : 0.f);
      }
    }
  };
  switch (kind) {
    case kRkEuler: finish(KindC<kRkEuler>{}); break;
    case kRk2Final: finish(KindC<kRk2Final>{}); break;
    case kRk3Mid: finish(KindC<kRk3Mid>{}); break;
    case kRk3Final: finish(KindC<kRk3Final>{}); break;
    default: finish(KindC<kRhsOnly>{}); break;
  }
  // the stability monitor (the last stage of a monitored step) reads the new
  // state back: this thread's own stores
  bool nonphys = false;
  if (P.monitor) {
    for (int k = 0; k < CPT; ++k) {
      const int e = tid + k * NT;
      if (e >= TX * TYE) break;
      const int tx = e % TX, ty = e / TX;
      const int gx = x0 + tx, gy = y0 + ty;
      if (gx >= nx || (ND > 1 && gy >= ny)) continue;
      const int64_t o = gy * P.sy + gx;
      double qn[S];
#pragma unroll
      for (int v = 0; v < S; ++v) qn[v] = qout[o + v * P.sv];
      double inv[ND];
      inv[0] = __ldg(P.inv_d[0] + gx);
      if constexpr (ND > 1) inv[1] = __ldg(P.inv_d[1] + gy);
      bool np;
      const double c = cell_icfl<ND, NF>(qn, P, dt, inv, np);
      nonphys |= np;
      if (!(c <= icfl)) icfl = c;  // keeps NaN
    }
  }
  if (bad && P.status) atomicOr(P.status, MFC_FLAG_NAN);
  if (nonphys && P.status) atomicOr(P.status, MFC_FLAG_NEG_PRESSURE);
  if (P.monitor) monitor_max(P.monitor, icfl);
}

template <int ND, int NF, int TX, int TY, int NT, bool GATE, bool VISC, int MINB, int RX, int RY>
__global__ void __launch_bounds__(NT, MINB) pair_kernel(const DevParams P, const __grid_constant__ UniformCoef U,
                                                        const double* __restrict__ qin,
                                                        const double* __restrict__ qbase, double* __restrict__ qout,
                                                        const double dt, const int kind, const PrimPairs B) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  pair_tile<ND, NF, TX, TY, NT, GATE, VISC, UniformCoef, false, RX, RY>(P, qin, qbase, qout, dt, kind, blockIdx.x * TX,
                                                                ND > 1 ? blockIdx.y * TY : 0, smem_raw, &U, B);
}

// With interior tiles loaded by TMA (2-D); T maps B.in or the stage input.
template <int NF, int TX, int TY, int NT, bool GATE, bool VISC, int MINB, int RX, int RY>
__global__ void __launch_bounds__(NT, MINB) pair_kernel_tma(const DevParams P, const __grid_constant__ UniformCoef U,
                                                            const __grid_constant__ TileMap T,
                                                            const double* __restrict__ qin,
                                                            const double* __restrict__ qbase,
                                                            double* __restrict__ qout, const double dt,
                                                            const int kind, const PrimPairs B) {
  extern __shared__ __align__(128) unsigned char smem_tma[];
  pair_tile<2, NF, TX, TY, NT, GATE, VISC, UniformCoef, true, RX, RY>(P, qin, qbase, qout, dt, kind, blockIdx.x * TX,
                                                               blockIdx.y * TY, smem_tma, &U, B, &T);
}

}  // namespace mfc
