// The fused RK-stage kernel: one launch computes, for a TX x TY tile of
// cells, everything MicroFC's s_compute_rhs does (m_rhs.fpp:405-679) and the
// RK stage update that follows it (m_time_steppers.fpp:298-348):
//
//   phase 1  load the tile plus an H-cell halo of the conservative state from
//            HBM (coalesced along x), apply the ghost-cell boundary conditions
//            by index mapping and convert to primitive variables in FP64
//   phase 2  x-direction WENO of every variable of every cell that borders a
//            face of the tile
//   phase 3  x-direction HLLC on the TX+1 faces of each row
//   phase 4  x flux divergence + alpha*div(u) into registers, and y WENO
//   phase 5  y-direction HLLC
//   phase 6  y flux divergence, RK combination, store (coalesced)
//
// Interface states and fluxes live only in shared memory; per stage HBM sees
// one read of the stage input (plus halo re-reads, which hit L2) and of the
// RK base register, and one write of the stage output.
#pragma once

#include <type_traits>

#include "mfc_device.cuh"
#include "mfc_tma.cuh"

namespace mfc {

// One cell's FP32 WENO coefficients from shared memory: kCoefRec floats,
// 16-byte aligned, as float4 loads.
template <class RT>
__device__ __forceinline__ void load_coef_record(const RT* __restrict__ rec, RT (&c)[kCoefRec]) {
  if constexpr (sizeof(RT) == 4) {
#pragma unroll
    for (int k = 0; k < kCoefRec / 4; ++k) {
      const float4 v = reinterpret_cast<const float4*>(rec)[k];
      c[4 * k] = v.x;
      c[4 * k + 1] = v.y;
      c[4 * k + 2] = v.z;
      c[4 * k + 3] = v.w;
    }
  }
}

// Precision changes of the accumulation type: identity for FP64, the
// integer bit-field conversions for the split path's FP32.
template <class T>
__device__ __forceinline__ T narrow(double x) {
  if constexpr (sizeof(T) == 4) return d2f_bits(x);
  else return x;
}
__device__ __forceinline__ double widen(double x) { return x; }
__device__ __forceinline__ double widen(float x) { return f2d_bits(x); }

template <int ND, int NF, int WO, class RT, int TX, int TY, bool VISC = false>
struct StageShape {
  using Q = Eqs<ND, NF>;
  static constexpr int S = Q::S;
  static constexpr int H = (WO + 1) / 2;  // halo depth
  static constexpr int TYE = (ND > 1) ? TY : 1;
  static constexpr int LX = TX + 2 * H;
  static constexpr int LY = (ND > 1) ? TY + 2 * H : 1;
  static constexpr int NQ = S * LY * LX;  // primitive tile
  // WENO outputs (left and right face values), x and y layouts share space
  static constexpr int NWX = S * TYE * (TX + 2);
  static constexpr int NWY = (ND > 1) ? S * (TY + 2) * TX : 0;
  static constexpr int NW = NWX > NWY ? NWX : NWY;
  // fluxes + interface velocity (+ the viscous x-momentum, y-momentum and
  // energy source fluxes)
  static constexpr int NR = S + 1 + (VISC ? 3 : 0);
  static constexpr int NFX = NR * TYE * (TX + 1);
  static constexpr int NFY = (ND > 1) ? NR * (TY + 1) * TX : 0;
  static constexpr int NFL = NFX > NFY ? NFX : NFY;
  static constexpr int NCX = TX + 2, NCY = (ND > 1) ? TY + 2 : 0;
  // FP64 WENO5: the tile's coefficients as doubles in [k][cell] order (x
  // cells, then y cells), staged once per tile so that the reconstructions
  // read them from shared memory instead of issuing kNumCoef global loads
  // each
  static constexpr int NCOEF = (sizeof(RT) == 8 && WO == 5) ? kNumCoef * (NCX + NCY) : 0;
  // offsets (in RT elements) of the arrays, each rounded up to 16 bytes
  static constexpr int align16(int n) { return (n * int(sizeof(RT)) + 15) / 16 * 16 / int(sizeof(RT)); }
  static constexpr int OW = align16(NQ), OF = OW + 2 * align16(NW), OC = OF + align16(NFL);
  // layout: primitive tile, WENO values, fluxes, coefficients
  static constexpr size_t kMainBytes = sizeof(RT) * size_t(OC);
  static constexpr size_t kCoefBytes = sizeof(RT) * size_t(NCOEF);
  static constexpr size_t kSmemBytes = kMainBytes + kCoefBytes;
};

// Where a tile finds the cell (rx, ry), inside the domain or up to H cells
// outside: the interior cell that a ghost cell mirrors (fx, fy: the normal
// momentum changes sign), or the halo buffer of a processor boundary.  vs:
// the stride between variables there.  Cells of partial edge tiles beyond the
// first H ghosts are never stored: their depth is clamped.  y strips are
// nx + 2 wide (the x ghost cells -1 and nx of the neighbour's rows come first
// and last).
template <int ND, int H>
__device__ __forceinline__ const double* tile_cell(const DevParams& P, const double* __restrict__ qin, const int rx,
                                                   const int ry, int64_t& vs, bool& fx, bool& fy) {
  const int nx = P.n[0], ny = P.n[1];
  fx = fy = false;
  vs = P.sv;
  const int px = rx < 0 ? (P.bc_beg[0] >= 0 ? 0 : -1) : (rx >= nx && P.bc_end[0] >= 0 ? 1 : -1);
  const int py = ND > 1 ? (ry < 0 ? (P.bc_beg[1] >= 0 ? 0 : -1) : (ry >= ny && P.bc_end[1] >= 0 ? 1 : -1)) : -1;
  if (px >= 0 && py >= 0) {
    // between two processor boundaries (the viscous corner cells): the
    // diagonal neighbour's cell, forwarded by the y neighbour
    const int d = min(py == 0 ? -1 - ry : ry - ny, H - 1);
    vs = (int64_t)H * (nx + 2);
    return P.halo[2 + py] + (int64_t)d * (nx + 2) + (px == 0 ? 0 : nx + 1);
  }
  if (px >= 0) {
    const int d = min(px == 0 ? -1 - rx : rx - nx, H - 1);
    const int yy = ND > 1 ? map_cell(ry, ny, P.bc_beg[1], P.bc_end[1], &fy) : 0;
    vs = (int64_t)ny * H;
    return P.halo[px] + (int64_t)yy * H + d;
  }
  if (py >= 0) {
    const int d = min(py == 0 ? -1 - ry : ry - ny, H - 1);
    const int xx = map_cell(rx, nx, P.bc_beg[0], P.bc_end[0], &fx);
    vs = (int64_t)H * (nx + 2);
    return P.halo[2 + py] + (int64_t)d * (nx + 2) + xx + 1;
  }
  const int gx = map_cell(rx, nx, P.bc_beg[0], P.bc_end[0], &fx);
  const int gy = ND > 1 ? map_cell(ry, ny, P.bc_beg[1], P.bc_end[1], &fy) : 0;
  return qin + gy * P.sy + gx;
}

// The TMA staging area of a stage tile (2-D): after the primitive tile,
// 128-byte aligned, the box of all variables, then its mbarrier and a flag.
template <int ND, int NF, int WO, class RT, int TX, int TY>
__device__ __forceinline__ unsigned char* tma_staging(unsigned char* smem_raw) {
  using Sh = StageShape<ND, NF, WO, RT, TX, TY>;
  const uintptr_t a = reinterpret_cast<uintptr_t>(smem_raw + Sh::OW * sizeof(RT));
  return reinterpret_cast<unsigned char*>((a + 127) & ~uintptr_t(127));
}
template <int ND, int NF, int WO, class RT, int TX, int TY>
constexpr uint32_t tma_stage_bytes() {
  using Sh = StageShape<ND, NF, WO, RT, TX, TY>;
  return uint32_t(TmaBox<TX, Sh::H>::kWidth) * Sh::LY * Sh::S * 8;
}

// Offset of the coefficients in a block's shared memory: after the main arrays
// and, in a TMA kernel, after the staging area (worst-case alignment), so that
// coefficients staged before the copy lands are not overwritten.
template <int ND, int NF, int WO, class RT, int TX, int TY, bool VISC, bool TMA>
constexpr size_t stage_coef_offset() {
  using Sh = StageShape<ND, NF, WO, RT, TX, TY, VISC>;
  size_t o = Sh::kMainBytes;
  if constexpr (TMA) {
    const size_t t =
        (sizeof(RT) * size_t(Sh::OW) + 128 + tma_stage_bytes<ND, NF, WO, RT, TX, TY>() + 16 + 15) / 16 * 16;
    o = o > t ? o : t;
  }
  return o;
}

// Dynamic shared memory of one block.
template <int ND, int NF, int WO, class RT, int TX, int TY, bool VISC, bool TMA>
constexpr size_t stage_smem_total() {
  return stage_coef_offset<ND, NF, WO, RT, TX, TY, VISC, TMA>() +
         StageShape<ND, NF, WO, RT, TX, TY, VISC>::kCoefBytes;
}

// WENO of the characteristic fields at one position (FP64): the stencil of
// the position's cell, at(v, o) = primitive variable v at offset o along DIR,
// is projected on the characteristic fields of the quasi-linear primitive
// system frozen at the cell's own state; each field is reconstructed with
// the cell's coefficients; the face values are mapped back to primitive
// variables into L(v) / R(v).  The fields (no counterpart in the
// reference, which reconstructs the primitive variables) in the slots of
// the primitive variables:
//   partial density i: alpha_i rho_i - kappa_i p,  kappa_i = alpha_i rho_i / (rho c^2)
//   normal momentum:   p - rho c u_n   (the u_n - c wave)
//   energy:            p + rho c u_n   (the u_n + c wave)
//   tangential velocities and volume fractions unchanged,
// with rho = max(sum alpha_i rho_i, 1e-16), Gamma = sum alpha_i Gamma_i,
// Pi = sum alpha_i Pi_i and c^2 = max(((Gamma + 1) p + Pi) / (Gamma rho),
// 1e-16), the mixture sound speed of the HLLC solver.  Back:
// p = (w+ + w-) 0.5, u_n = (w+ - w-) / (2 rho c), alpha_i rho_i = w_i + kappa_i p.
// The oracle (Solver::weno with char_decomp) evaluates the same expressions
// in the same order.
template <int ND, int NF, int WO, int DIR, class At, class OutL, class OutR>
__device__ __forceinline__ void char_weno_position(const double (&c)[kCoefRec], const At& at, const double eps,
                                                   const DevParams& P, const Num64& u0, const OutL& L, const OutR& R) {
  using Q = Eqs<ND, NF>;
  constexpr int S = Q::S, UN = Q::MOM + DIR;
  double rho = 0.0, gam = 0.0, pinf = 0.0;
#pragma unroll
  for (int f = 0; f < NF; ++f) {
    rho = rho + at(f, 0);
    gam = gam + at(Q::ADV + f, 0) * P.gammas[f];
    pinf = pinf + at(Q::ADV + f, 0) * P.pi_infs[f];
  }
  rho = fmax(rho, 1e-16);
  const double c2 = fmax(div_rn((gam + 1.0) * at(Q::E, 0) + pinf, divisor(gam * rho)), 1e-16);
  const double rc = rho * sqrt(c2);
  const DivisorF64 Dk = divisor(rho * c2);
  double kap[NF];
#pragma unroll
  for (int f = 0; f < NF; ++f) kap[f] = div_rn(at(f, 0), Dk);
#pragma unroll 1
  for (int v = 0; v < S; ++v) {
    double st[5];
#pragma unroll
    for (int k = 0; k < 5; ++k) {
      const int o = k - 2;
      if (o < -(WO / 2) || o > WO / 2) {
        st[k] = 0.0;
      } else if (v < NF) {
        double kv = kap[0];
#pragma unroll
        for (int f = 1; f < NF; ++f) kv = v == f ? kap[f] : kv;
        st[k] = at(v, o) - kv * at(Q::E, o);
      } else if (v == UN) {
        st[k] = at(Q::E, o) - rc * at(UN, o);
      } else if (v == Q::E) {
        st[k] = at(Q::E, o) + rc * at(UN, o);
      } else {
        st[k] = at(v, o);
      }
    }
    Num64 ns[5], vl, vr;
#pragma unroll
    for (int k = 0; k < 5; ++k) ns[k] = lift(st[k], u0);
    weno_cell<WO, Num64>(NumCoef<Num64>{c, u0}, ns, lift(eps, u0), vl, vr);
    L(v) = low(vl);
    R(v) = low(vr);
  }
  const DivisorF64 D2 = divisor(2.0 * rc);
  auto back = [&](const auto& O) {
    const double wm = O(UN), wp = O(Q::E);
    const double pr = (wp + wm) * 0.5;
    O(Q::E) = pr;
    O(UN) = div_rn(wp - wm, D2);
#pragma unroll
    for (int f = 0; f < NF; ++f) O(f) = O(f) + kap[f] * pr;
  };
  back(L);
  back(R);
}

// One tile of one RK stage; the tile's first cell is (x0, y0).  Used by the
// single-case kernel and by the FP64 ensemble kernel.  smem_raw must hold
// stage_smem_total().
template <int ND, int NF, int WO, class RT, int TX, int TY, int NT, bool VISC = false, bool TMA = false,
          bool CHAR = false>
__device__ __forceinline__ void stage_tile(const DevParams& P, const double* __restrict__ qin,
                                           const double* __restrict__ qbase, double* __restrict__ qout,
                                           const double dt, const int kind, const int x0, const int y0,
                                           unsigned char* smem_raw, const TileMap* T = nullptr) {
  static_assert(sizeof(RT) == 8 || WO < 5, "split-precision WENO5 is pair_tile (mfc_pair.cuh)");
  static_assert(!CHAR || (sizeof(RT) == 8 && WO > 1 && !VISC && ND < 3),
                "characteristic-field WENO is compiled for the inviscid FP64 1-D/2-D WENO3/5 kernel");
  using Sh = StageShape<ND, NF, WO, RT, TX, TY, VISC>;
  using Q = Eqs<ND, NF>;
  constexpr int S = Sh::S, H = Sh::H, LX = Sh::LX, LY = Sh::LY, TYE = Sh::TYE;
  constexpr int CPT = (TX * TYE + NT - 1) / NT;  // interior cells per thread
  // split precision: FP32 reconstruction, Riemann solve and flux divergence;
  // the plain path keeps everything in FP64 in the reference's order
  constexpr bool kSplit = sizeof(RT) == 4;
  using AT = RT;  // storage of the flux-divergence accumulation
  // what the arithmetic runs on (Fma64 for the plain path)
  using N = std::conditional_t<kSplit, float, Num64>;
  N u0;
  if constexpr (kSplit) u0 = 0.f;
  else u0 = num64_unit(P.inv_d[0]);
  auto num = [&](RT x) { return lift(x, u0); };
  // split: the FP64 sums' register operand (1-D: a constant; loading it cost
  // 30.4 against 28.9 us a step at 1000 cells, WENO3)
  const double one = kSplit && ND > 1 ? fma64_unit(P.inv_d[0]).one : 1.0;
  (void)one;

  RT* sq = reinterpret_cast<RT*>(smem_raw);  // [S][LY][LX] primitive
  RT* wl = sq + Sh::OW;                       // left-face values
  RT* wr = wl + Sh::align16(Sh::NW);          // right-face values
  RT* fl = sq + Sh::OF;                       // fluxes [S+1][...]
  // FP64 WENO5: coefficients [kNumCoef][TX+2], then [kNumCoef][TY+2]
  RT* scx = reinterpret_cast<RT*>(smem_raw + stage_coef_offset<ND, NF, WO, RT, TX, TY, VISC, TMA>());
  RT* scy = scx + kNumCoef * Sh::NCX;
  // element of variable v in the primitive tile and in the x / y WENO values
  auto qi = [](int v, int ly, int lx) { return (v * LY + ly) * LX + lx; };
  auto wxi = [](int v, int ty, int cx) { return (v * TYE + ty) * Sh::NCX + cx; };
  auto wyi = [](int v, int cy, int tx) { return (v * Sh::NCY + cy) * TX + tx; };
  (void)scy;
  (void)wyi;
  // row r of the flux of x face f (left of cell f) of row ty, and of y face f
  auto fxv = [&](int r, int ty, int f) -> RT& { return fl[(r * TYE + ty) * (TX + 1) + f]; };
  auto fyv = [&](int r, int f, int tx) -> RT& { return fl[(r * (TY + 1) + f) * TX + tx]; };
  (void)fyv;

  const int tid = threadIdx.x;
  const int nx = P.n[0], ny = P.n[1];

  N gam_i[NF], pi_i[NF];
#pragma unroll
  for (int f = 0; f < NF; ++f) {
    if constexpr (kSplit) {
      gam_i[f] = P.gammas_f[f];
      pi_i[f] = P.pi_infs_f[f];
    } else {
      gam_i[f] = num(P.gammas[f]);
      pi_i[f] = num(P.pi_infs[f]);
    }
  }
  N eps;
  if constexpr (kSplit) eps = P.weno_eps_f;
  else eps = num(P.weno_eps);
  // ---- phase 1: load + BCs + cons -> prim --------------------------------
  if constexpr (Sh::NCOEF > 0 && !CHAR) {
    // FP64 WENO5: the tile's coefficients, [k][cell], before the wait
    for (int it = tid; it < kNumCoef * Sh::NCX; it += NT) {
      const int cx = it % Sh::NCX, k = it / Sh::NCX;
      scx[k * Sh::NCX + cx] = __ldg(P.coef[0] + k * P.cstride[0] + clamp_coef_index(x0 - 1 + cx, nx) + P.coff);
    }
    if constexpr (ND > 1) {
      for (int it = tid; it < kNumCoef * Sh::NCY; it += NT) {
        const int cy = it % Sh::NCY, k = it / Sh::NCY;
        scy[k * Sh::NCY + cy] = __ldg(P.coef[1] + k * P.cstride[1] + clamp_coef_index(y0 - 1 + cy, ny) + P.coff);
      }
    }
  }
  // one cell of the tile: BCs already applied, cons -> prim into the tile
  auto store_prim = [&](double (&q)[S], const int ly, const int lx) {
    if constexpr (kSplit) {
      float pr[S];
      cons_to_prim_split<ND, NF>(q, P, one, pr);
#pragma unroll
      for (int v = 0; v < S; ++v) sq[qi(v, ly, lx)] = pr[v];
    } else {
      cons_to_prim<ND, NF>(q, P, u0);
#pragma unroll
      for (int v = 0; v < S; ++v) sq[qi(v, ly, lx)] = RT(q[v]);
    }
  };
  // corners are never read, except the four diagonal neighbours of the tile
  // that the viscous cross derivatives use
  auto unused_corner = [](const int lx, const int ly) {
    const bool hx = lx < H || lx >= H + TX;
    const bool hy = (ND > 1) && (ly < H || ly >= H + TY);
    return hx && hy && !(VISC && (lx == H - 1 || lx == H + TX) && (ly == H - 1 || ly == H + TY));
  };

  // TMA staging: a tile whose halo lies inside the domain (no boundary
  // condition, no processor halo) arrives in one bulk tensor copy of all
  // variables into the WENO and flux arrays, which are free until phase 2
  // (the coefficients sit past the staging area).
  bool use_tma = false;
  unsigned char* stg = nullptr;
  uint32_t bar = 0;
  using Box = TmaBox<TX, H>;
  constexpr uint32_t kStageBytes = tma_stage_bytes<ND, NF, WO, RT, TX, TY>();
  if constexpr (TMA && ND == 2 && !VISC) {
    use_tma = T != nullptr && T->on && x0 >= H && x0 + TX + H <= nx && y0 >= H && y0 + TY + H <= ny;
    if (use_tma) {
      stg = tma_staging<ND, NF, WO, RT, TX, TY>(smem_raw);
      bar = smem_addr(stg + kStageBytes);
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
      const int gx = x0 + line * 16, gy = (ND > 1) ? y0 + ty : 0;
      if (gx >= nx || gy >= ny) continue;
      asm volatile("prefetch.global.L2 [%0];" ::"l"(qbase + gy * P.sy + gx + v * P.sv));
    }
  }
  if (use_tma) {
    volatile int* landed = reinterpret_cast<volatile int*>(stg + kStageBytes + 8);
    if (tid == 0) {
      mbar_arrive_expect_tx(bar, kStageBytes);
      tma_load_3d(smem_addr(stg), &T->map, x0 - Box::kLead, y0 - H, 0, bar);
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
    for (int c = tid; c < LX * LY; c += NT) {
      const int lx = c % LX, ly = c / LX;
      if (unused_corner(lx, ly)) continue;
      double q[S];
#pragma unroll
      for (int v = 0; v < S; ++v) q[v] = sd[(v * LY + ly) * Box::kWidth + lx + (Box::kLead - H)];
      store_prim(q, ly, lx);
    }
  } else {  // plain loads, with the boundary conditions and processor halos
    for (int c = tid; c < LX * LY; c += NT) {
      const int lx = c % LX, ly = c / LX;
      if (unused_corner(lx, ly)) continue;
      bool fx, fy;
      int64_t vs;
      const double* src = tile_cell<ND, H>(P, qin, x0 - H + lx, ND > 1 ? y0 - H + ly : 0, vs, fx, fy);
      double q[S];
#pragma unroll
      for (int v = 0; v < S; ++v) q[v] = __ldg(src + v * vs);
      if (fx) q[Q::MOM] = -q[Q::MOM];
      if (ND > 1 && fy) q[Q::MOM + 1] = -q[Q::MOM + 1];
      store_prim(q, ly, lx);
    }
  }
  __syncthreads();

  // ---- phase 2: x WENO over cells x0-1 .. x0+TX of the interior rows -------
  {
    constexpr int NCX = TX + 2;
    // variable v of the cell at (cx, ty); c: the cell's coefficient record
    auto x_recon = [&](const RT* __restrict__ c, const int cx, const int ty, const int v) {
      N st[5];
#pragma unroll
      for (int k = 0; k < 5; ++k) {
        const int o = k - 2;
        st[k] = num(o >= -(WO / 2) && o <= WO / 2 ? sq[qi(v, (ND > 1) ? ty + H : 0, cx + H - 1 + o)] : RT(0));
      }
      N vl, vr;
      if constexpr (kSplit) weno_cell<WO, N>(c, st, eps, vl, vr);
      else weno_cell<WO, N>(NumCoef<N>{c, u0}, st, eps, vl, vr);
      wl[wxi(v, ty, cx)] = low(vl);
      wr[wxi(v, ty, cx)] = low(vr);
    };
    if constexpr (CHAR) {
      // characteristic fields: one thread per position, all variables
      const double* cf = P.coef[0];
      const int cs = P.cstride[0];
      for (int it = tid; it < TYE * NCX; it += NT) {
        const int cx = it % NCX, ty = it / NCX;
        RT c[kCoefRec];
        const int gi = clamp_coef_index(x0 - 1 + cx, nx) + P.coff;
#pragma unroll
        for (int k = 0; k < kNumCoef; ++k) c[k] = RT(__ldg(cf + k * cs + gi));
        const int ly = (ND > 1) ? ty + H : 0, lx = cx + H - 1;
        char_weno_position<ND, NF, WO, 0>(
            c, [&](int v, int o) { return sq[qi(v, ly, lx + o)]; }, low(eps), P, u0,
            [&](int v) -> RT& { return wl[wxi(v, ty, cx)]; }, [&](int v) -> RT& { return wr[wxi(v, ty, cx)]; });
      }
    } else if constexpr (sizeof(RT) == 8 && WO > 1) {
      // FP64: positions cx = 1 .. TX feed two faces each; the tile-edge
      // positions feed one -- cell x0 - 1 only its right-face value (the left
      // state of face x0 - 1/2), cell x0 + TX only its left-face value -- so
      // only that value is formed there (weno_cell_side, the same bits).  The
      // edge items go to the threads that have one interior item fewer.
      // the tile's staged coefficients (WENO3: from global memory)
      const double* cf = P.coef[0];
      const int cs = P.cstride[0];
      auto coef = [&](const int cx, RT (&c)[kCoefRec]) {
        if constexpr (Sh::NCOEF > 0) {
#pragma unroll
          for (int k = 0; k < kNumCoef; ++k) c[k] = scx[k * Sh::NCX + cx];
        } else {
          const int gi = clamp_coef_index(x0 - 1 + cx, nx) + P.coff;
#pragma unroll
          for (int k = 0; k < kNumCoef; ++k) c[k] = RT(__ldg(cf + k * cs + gi));
        }
      };
      constexpr int NI = S * TYE * TX, NE = S * TYE * 2;
      for (int it = tid; it < NI; it += NT) {
        const int cx = 1 + it % TX, r = it / TX;
        const int ty = r % TYE, v = r / TYE;
        RT c[kCoefRec];
        coef(cx, c);
        x_recon(c, cx, ty, v);
      }
      for (int it = (tid + NT - NI % NT) % NT; it < NE; it += NT) {
        const int side = it / (S * TYE), r = it % (S * TYE);
        const int ty = r % TYE, v = r / TYE, cx = side ? NCX - 1 : 0;
        RT c[kCoefRec];
        coef(cx, c);
        N st[5];
#pragma unroll
        for (int k = 0; k < 5; ++k) {
          const int o = k - 2;
          st[k] = num(o >= -(WO / 2) && o <= WO / 2 ? sq[qi(v, (ND > 1) ? ty + H : 0, cx + H - 1 + o)] : RT(0));
        }
        if (side) wl[wxi(v, ty, cx)] = low(weno_cell_side<WO, 0, N>(NumCoef<N>{c, u0}, st, eps));
        else wr[wxi(v, ty, cx)] = low(weno_cell_side<WO, 1, N>(NumCoef<N>{c, u0}, st, eps));
      }
    } else {
      // split WENO1/3 and FP64 WENO1: coefficients per reconstruction from global memory
      const double* cf = P.coef[0];
      const int cs = P.cstride[0];
      for (int it = tid; it < S * TYE * NCX; it += NT) {
        const int cx = it % NCX;
        const int r = it / NCX;
        const int ty = r % TYE, v = r / TYE;
        RT c[kCoefRec];
        if constexpr (WO > 1) {
          const int gi = clamp_coef_index(x0 - 1 + cx, nx) + P.coff;
#pragma unroll
          for (int k = 0; k < kNumCoef; ++k) c[k] = RT(__ldg(cf + k * cs + gi));
        }
        x_recon(c, cx, ty, v);
      }
    }
  }
  __syncthreads();

  // ---- phase 3: x HLLC on faces x0-1/2 .. x0+TX-1/2 ------------------------
  {
    constexpr int NFXr = TX + 1;
    for (int it = tid; it < TYE * NFXr; it += NT) {
      const int f = it % NFXr, ty = it / NFXr;
      const int gface = x0 - 1 + f;  // face gface+1/2
      N qL[S], qR[S], F[S], us;
      const bool lfr = (gface == -1 && P.bc_beg[0] == -4);      // qL(-1) = qR(0)
      const bool rfl = (gface == nx - 1 && P.bc_end[0] == -4);  // qR(m+1) = qL(m)
#pragma unroll
      for (int v = 0; v < S; ++v) {
        const N a = num(wr[wxi(v, ty, f)]);
        const N b = num(wl[wxi(v, ty, f + 1)]);
        qL[v] = lfr ? b : a;
        qR[v] = rfl ? a : b;
      }
      if constexpr (VISC) {
        N vs[ND], dxv[2] = {num(RT(0)), num(RT(0))}, dyv[2] = {num(RT(0)), num(RT(0))}, vf[3];
        hllc_face<ND, NF, 0, N, true>(qL, qR, gam_i, pi_i, F, us, vs);
        const ViscParams& V = *P.visc;
        const int ly = (ND > 1) ? ty + H : 0, lx = f + H - 1;  // the face's left cell
        auto U = [&](int c, int x, int y) { return num(sq[qi(Q::MOM + c, y, x)]); };
        const auto Dx = divisor(narrow<RT>(__ldg(V.dcc[0] + min(x0 + f, nx))));  // x_cc(j+1) - x_cc(j)
#pragma unroll
        for (int c = 0; c < ND; ++c) {
          const N g = div_rn(U(c, lx + 1, ly) - U(c, lx, ly), Dx);
          dxv[c] = num(RT(0.5)) * (g + g);
        }
        if constexpr (ND > 1) {
          const int gy = min(y0 + ty, ny - 1);
          const auto D0 = divisor(narrow<RT>(__ldg(V.dcc[1] + gy))),
                     D1 = divisor(narrow<RT>(__ldg(V.dcc[1] + gy + 1)));
#pragma unroll
          for (int c = 0; c < ND; ++c) {
            auto Ly = [&](int x) { return div_rn(U(c, x, ly) - U(c, x, ly - 1), D0); };
            auto Ry = [&](int x) { return div_rn(U(c, x, ly + 1) - U(c, x, ly), D1); };
            const N A = num(RT(0.25)) * (Ly(lx + 1) + Ry(lx + 1) + Ly(lx) + Ry(lx));
            dyv[c] = num(RT(0.5)) * (A + A);
          }
        }
        viscous_face_flux<ND, NF, 0, N>(qL, qR, V, vs, dxv, dyv, vf);
#pragma unroll
        for (int t = 0; t < 3; ++t) fxv(S + 1 + t, ty, f) = low(vf[t]);
      } else if constexpr (kSplit) {
        hllc_face_fast<ND, NF, 0>(qL, qR, gam_i, pi_i, F, us);
      } else {
        hllc_face<ND, NF, 0, N>(qL, qR, gam_i, pi_i, F, us);
      }
#pragma unroll
      for (int v = 0; v < S; ++v) fxv(v, ty, f) = low(F[v]);
      fxv(S, ty, f) = low(us);
    }
  }
  __syncthreads();

  // ---- phase 4: x flux divergence (registers) + y WENO ----------------------
  AT rhs[CPT][S];
#pragma unroll
  for (int k = 0; k < CPT; ++k) {
    const int e = tid + k * NT;
    if (e >= TX * TYE) break;
    const int tx = e % TX, ty = e / TX;
    const int gx = x0 + tx;
    const N inv = num(narrow<AT>(__ldg(P.inv_d[0] + (gx < nx ? gx : nx - 1))));
#pragma unroll
    for (int v = 0; v < S; ++v) rhs[k][v] = low(inv * (num(fxv(v, ty, tx)) - num(fxv(v, ty, tx + 1))));
    const N du = num(fxv(S, ty, tx + 1)) - num(fxv(S, ty, tx));
#pragma unroll
    for (int f = 0; f < NF; ++f) {
      const N a = num(sq[qi(Q::ADV + f, ND > 1 ? ty + H : 0, tx + H)]);
      rhs[k][Q::ADV + f] = low(mul_add(inv * a, du, num(rhs[k][Q::ADV + f])));
    }
    if constexpr (VISC) {  // m_rhs.fpp:591-603: momentum .. energy
#pragma unroll
      for (int t = 0; t <= ND; ++t) {
        const int v = t < ND ? Q::MOM + t : Q::E, r = S + 1 + (t < ND ? t : 2);
        rhs[k][v] = low(mul_add(inv, num(fxv(r, ty, tx)) - num(fxv(r, ty, tx + 1)), num(rhs[k][v])));
      }
    }
  }
  if constexpr (ND > 1) {
    constexpr int NCY = TY + 2;
    // variable v of the cell at (tx, cy)
    auto y_recon = [&](const RT* __restrict__ c, const int tx, const int cy, const int v) {
      N st[5];
#pragma unroll
      for (int k = 0; k < 5; ++k) {
        const int o = k - 2;
        st[k] = num(o >= -(WO / 2) && o <= WO / 2 ? sq[qi(v, cy + H - 1 + o, tx + H)] : RT(0));
      }
      N vl, vr;
      if constexpr (kSplit) weno_cell<WO, N>(c, st, eps, vl, vr);
      else weno_cell<WO, N>(NumCoef<N>{c, u0}, st, eps, vl, vr);
      wl[wyi(v, cy, tx)] = low(vl);
      wr[wyi(v, cy, tx)] = low(vr);
    };
    if constexpr (CHAR) {
      const double* cf = P.coef[1];
      const int cs = P.cstride[1];
      for (int it = tid; it < NCY * TX; it += NT) {
        const int tx = it % TX, cy = it / TX;
        RT c[kCoefRec];
        const int gi = clamp_coef_index(y0 - 1 + cy, ny) + P.coff;
#pragma unroll
        for (int k = 0; k < kNumCoef; ++k) c[k] = RT(__ldg(cf + k * cs + gi));
        const int ly = cy + H - 1, lx = tx + H;
        char_weno_position<ND, NF, WO, 1>(
            c, [&](int v, int o) { return sq[qi(v, ly + o, lx)]; }, low(eps), P, u0,
            [&](int v) -> RT& { return wl[wyi(v, cy, tx)]; }, [&](int v) -> RT& { return wr[wyi(v, cy, tx)]; });
      }
    } else if constexpr (sizeof(RT) == 8 && WO > 1) {
      // FP64: rows cy = 1 .. TY feed two faces each; row y0 - 1 only its
      // upper-face value, row y0 + TY only its lower-face value (as in x)
      const double* cf = P.coef[1];
      const int cs = P.cstride[1];
      auto coef = [&](const int cy, RT (&c)[kCoefRec]) {
        if constexpr (Sh::NCOEF > 0) {
#pragma unroll
          for (int k = 0; k < kNumCoef; ++k) c[k] = scy[k * Sh::NCY + cy];
        } else {
          const int gi = clamp_coef_index(y0 - 1 + cy, ny) + P.coff;
#pragma unroll
          for (int k = 0; k < kNumCoef; ++k) c[k] = RT(__ldg(cf + k * cs + gi));
        }
      };
      constexpr int NI = S * TY * TX, NE = S * 2 * TX;
      for (int it = tid; it < NI; it += NT) {
        const int tx = it % TX, r = it / TX;
        const int cy = 1 + r % TY, v = r / TY;
        RT c[kCoefRec];
        coef(cy, c);
        y_recon(c, tx, cy, v);
      }
      for (int it = (tid + NT - NI % NT) % NT; it < NE; it += NT) {
        const int side = it / (S * TX), r = it % (S * TX);
        const int tx = r % TX, v = r / TX, cy = side ? NCY - 1 : 0;
        RT c[kCoefRec];
        coef(cy, c);
        N st[5];
#pragma unroll
        for (int k = 0; k < 5; ++k) {
          const int o = k - 2;
          st[k] = num(o >= -(WO / 2) && o <= WO / 2 ? sq[qi(v, cy + H - 1 + o, tx + H)] : RT(0));
        }
        if (side) wl[wyi(v, cy, tx)] = low(weno_cell_side<WO, 0, N>(NumCoef<N>{c, u0}, st, eps));
        else wr[wyi(v, cy, tx)] = low(weno_cell_side<WO, 1, N>(NumCoef<N>{c, u0}, st, eps));
      }
    } else {
      const double* cf = P.coef[1];
      const int cs = P.cstride[1];
      for (int it = tid; it < S * NCY * TX; it += NT) {
        const int tx = it % TX;
        const int r = it / TX;
        const int cy = r % NCY, v = r / NCY;
        RT c[kCoefRec];
        if constexpr (WO > 1) {
          const int gi = clamp_coef_index(y0 - 1 + cy, ny) + P.coff;
#pragma unroll
          for (int k = 0; k < kNumCoef; ++k) c[k] = RT(__ldg(cf + k * cs + gi));
        }
        y_recon(c, tx, cy, v);
      }
    }
    __syncthreads();

    // ---- phase 5: y HLLC on faces y0-1/2 .. y0+TY-1/2 ----------------------
    constexpr int NFYr = TY + 1;
    for (int it = tid; it < NFYr * TX; it += NT) {
      const int tx = it % TX, f = it / TX;
      const int gface = y0 - 1 + f;
      N qL[S], qR[S], F[S], us;
      const bool lfr = (gface == -1 && P.bc_beg[1] == -4);
      const bool rfl = (gface == ny - 1 && P.bc_end[1] == -4);
#pragma unroll
      for (int v = 0; v < S; ++v) {
        const N a = num(wr[wyi(v, f, tx)]);
        const N b = num(wl[wyi(v, f + 1, tx)]);
        qL[v] = lfr ? b : a;
        qR[v] = rfl ? a : b;
      }
      if constexpr (VISC) {
        N vs[ND], dxv[2], dyv[2], vf[3];
        hllc_face<ND, NF, 1, N, true>(qL, qR, gam_i, pi_i, F, us, vs);
        const ViscParams& V = *P.visc;
        const int gx = min(x0 + tx, nx - 1);
        const int ly = f + H - 1, lx = tx + H;  // the face's lower cell
        auto U = [&](int c, int x, int y) { return num(sq[qi(Q::MOM + c, y, x)]); };
        const auto Dy = divisor(narrow<RT>(__ldg(V.dcc[1] + min(y0 + f, ny))));  // y_cc(k+1) - y_cc(k)
        const auto D0 = divisor(narrow<RT>(__ldg(V.dcc[0] + gx))),
                   D1 = divisor(narrow<RT>(__ldg(V.dcc[0] + gx + 1)));
#pragma unroll
        for (int c = 0; c < 2; ++c) {
          auto Lx = [&](int y) { return div_rn(U(c, lx, y) - U(c, lx - 1, y), D0); };
          auto Rx = [&](int y) { return div_rn(U(c, lx + 1, y) - U(c, lx, y), D1); };
          const N A = num(RT(0.25)) * (Lx(ly + 1) + Rx(ly + 1) + Lx(ly) + Rx(ly));
          dxv[c] = num(RT(0.5)) * (A + A);
          const N g = div_rn(U(c, lx, ly + 1) - U(c, lx, ly), Dy);
          dyv[c] = num(RT(0.5)) * (g + g);
        }
        viscous_face_flux<ND, NF, 1, N>(qL, qR, V, vs, dxv, dyv, vf);
#pragma unroll
        for (int t = 0; t < 3; ++t) fyv(S + 1 + t, f, tx) = low(vf[t]);
      } else if constexpr (kSplit) {
        hllc_face_fast<ND, NF, 1>(qL, qR, gam_i, pi_i, F, us);
      } else {
        hllc_face<ND, NF, 1, N>(qL, qR, gam_i, pi_i, F, us);
      }
#pragma unroll
      for (int v = 0; v < S; ++v) fyv(v, f, tx) = low(F[v]);
      fyv(S, f, tx) = low(us);
    }
    __syncthreads();

    // ---- phase 6a: y flux divergence ------------------------------------------
#pragma unroll
    for (int k = 0; k < CPT; ++k) {
      const int e = tid + k * NT;
      if (e >= TX * TY) break;
      const int tx = e % TX, ty = e / TX;
      const int gy = y0 + ty;
      const N inv = num(narrow<AT>(__ldg(P.inv_d[1] + (gy < ny ? gy : ny - 1))));
#pragma unroll
      for (int v = 0; v < S; ++v)
        rhs[k][v] = low(mul_add(inv, num(fyv(v, ty, tx)) - num(fyv(v, ty + 1, tx)), num(rhs[k][v])));
      const N du = num(fyv(S, ty + 1, tx)) - num(fyv(S, ty, tx));
#pragma unroll
      for (int f = 0; f < NF; ++f) {
        const N a = num(sq[qi(Q::ADV + f, ty + H, tx + H)]);
        rhs[k][Q::ADV + f] = low(mul_add(inv * a, du, num(rhs[k][Q::ADV + f])));
      }
      if constexpr (VISC) {  // m_rhs.fpp:639-651
#pragma unroll
        for (int t = 0; t <= ND; ++t) {
          const int v = t < ND ? Q::MOM + t : Q::E, r = S + 1 + (t < ND ? t : 2);
          rhs[k][v] = low(mul_add(inv, num(fyv(r, ty, tx)) - num(fyv(r, ty + 1, tx)), num(rhs[k][v])));
        }
      }
    }
  }

  // ---- phase 6b: RK combination and store ------------------------------------
  griddep_launch_dependents();
  bool bad = false;
  const float dtf = kSplit ? __double2float_rn(dt) : 0.f;  // the split path's increments are FP32
  (void)dtf;
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
#pragma unroll
      for (int v = 0; v < S; ++v) {
        double out;
        if constexpr (KIND == kRhsOnly) {
          out = widen(rhs[k][v]);
        } else {
          const double b = __ldg(qbase + o + v * P.sv);
          double in = b;
          if constexpr (KIND != kRkEuler) in = __ldg(qin + o + v * P.sv);
          if constexpr (kSplit) out = rk_combine_split(KIND, b, in, dtf, rhs[k][v], one);
          else out = rk_combine(KIND, num(b), num(in), num(dt), num(rhs[k][v]));
        }
        bad |= not_finite(out);
        qout[o + v * P.sv] = out;
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

// FMA tags the instantiations of the translation unit compiled with
// multiply-add contraction (-fmad=true), so that their host-side symbols
// differ from the bit-faithful ones; the kernel body does not use it.
template <int ND, int NF, int WO, class RT, int TX, int TY, int NT, bool FMA = false, bool CHAR = false>
__global__ void __launch_bounds__(NT) stage_kernel(const DevParams P, const double* __restrict__ qin,
                                                   const double* __restrict__ qbase, double* __restrict__ qout,
                                                   const double dt, const int kind) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  stage_tile<ND, NF, WO, RT, TX, TY, NT, false, false, CHAR>(P, qin, qbase, qout, dt, kind, blockIdx.x * TX,
                                                             (ND > 1) ? blockIdx.y * TY : 0, smem_raw);
}

// The kernel with TMA staging of interior tiles (2-D, inviscid); T maps the
// stage input qin.
template <int ND, int NF, int WO, class RT, int TX, int TY, int NT, bool FMA = false>
__global__ void __launch_bounds__(NT) stage_kernel_tma(const DevParams P, const __grid_constant__ TileMap T,
                                                       const double* __restrict__ qin,
                                                       const double* __restrict__ qbase, double* __restrict__ qout,
                                                       const double dt, const int kind) {
  extern __shared__ __align__(128) unsigned char smem_tma[];
  stage_tile<ND, NF, WO, RT, TX, TY, NT, false, true>(P, qin, qbase, qout, dt, kind, blockIdx.x * TX,
                                                      (ND > 1) ? blockIdx.y * TY : 0, smem_tma, &T);
}

}  // namespace mfc
