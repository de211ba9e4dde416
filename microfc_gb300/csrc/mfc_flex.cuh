// The plain FP64 RK stage of 1-D and 2-D cases on tiles whose size is chosen
// at run time: the work of stage_tile (mfc_stage.cuh), the same operations in
// the same order on the same number type, hence the same bits, split so that
// every SM gets an equal share of the grid.
//
// What bounds it: the SM's FP64 unit (one warp operation per 16 cycles;
// about 680 of them per direction for 32 cells), everything else hides
// behind it.  So the time of a stage is the largest number of FP64
// operations any SM has to do, and a fixed tile loses by rounding: 400x200
// cells are 169 tiles of 32x16, two waves on 152 SMs.  Here a grid of any
// size is cut into a multiple of 152 nearly equal tiles (flex_plan), the
// partial tiles at the upper edges do no work for cells outside the domain,
// and both directions go through each phase together:
//
//   load + BCs + cons -> prim | WENO x and y | HLLC x and y | divergence + RK
//
// Half the barriers of the x-then-y order, and twice the warp items between
// them, so that small tiles keep four warps (what the FP64 unit needs) busy.
// The items of a phase are dealt to the warps 32 at a time, one direction
// and kind per group.  A face's flux overwrites the two states that it was
// solved from (the right value of the cell before it, the left value of the
// cell after it: no other face reads either), so there is no flux array.
//
// Measured (us a step, before: the default fixed tile, 32x16 or, viscous,
// 16x16 and in 1-D 128 cells): 100x100 632 -> 118, 301x101 634 -> 272,
// 400x200 1225 -> 647, 1024x512 4293 -> 4008, 2048x1024 16552 -> 15761,
// viscous 320x160 871 -> 526, 1-D 1000 cells 140 -> 42 (with hllc_face's
// later form 263, 620, 3848, 522 and 38, and in 1-D, with
// flex_sides and flex_lane_pairs, 29.5).  640 threads (96
// registers) against 512 (114): 4008 and 4093 at 1024x512; the viscous
// kernel, whose faces need the registers, is faster with 512.
#pragma once

#include "mfc_device.cuh"
#include "mfc_stage.cuh"
#include "mfc_sweep.cuh"

namespace mfc {

constexpr size_t kFlexSmemMax = 227 * 1024;

// Shared memory of a tx x ty tile, in doubles: primitives with their halo,
// the left and right WENO values of each direction, the WENO coefficients.
template <int ND, int NF, int WO>
struct FlexShape {
  static constexpr int S = Eqs<ND, NF>::S, H = (WO + 1) / 2;
  __host__ __device__ static int nq(int tx, int ty) { return S * (tx + 2 * H) * (ND > 1 ? ty + 2 * H : 1); }
  __host__ __device__ static int nwx(int tx, int ty) { return S * (tx + 2) * ty; }
  __host__ __device__ static int nwy(int tx, int ty) { return ND > 1 ? S * (ty + 2) * tx : 0; }
  __host__ __device__ static int ncoef(int tx, int ty) {
    return WO > 1 ? kNumCoef * (tx + 2 + (ND > 1 ? ty + 2 : 0)) : 0;
  }
  static size_t bytes(int tx, int ty) {
    return sizeof(double) * ((size_t)nq(tx, ty) + 2 * (size_t)nwx(tx, ty) + 2 * (size_t)nwy(tx, ty) +
                             (size_t)ncoef(tx, ty));
  }
};

// The phases of small 1-D tiles, whose few warps are bound by their chains (64
// cycles an operation) and not by the FP64 unit (16.5 a warp operation): a
// reconstruction's two face values go to two items (53 operations each in
// place of 72 for both) and a face's two states to two lanes (59 operations
// deep in place of 85) where that is the shorter of the two bounds.  gi, ge:
// groups of interior and of end positions, gs: groups of one side's values.
// us a step without and with both: 300 cells 36.1 -> 28.8, 1000 38.1 -> 29.5,
// 4000 44.0 -> 41.0; 20000, which take neither, 103.4 and 104.1.
template <int WO>
__host__ __device__ inline bool flex_sides(int gi, int ge, int gs, int warps) {
  constexpr float both = WO == 5 ? 72.f : 26.f, one = WO == 5 ? 53.f : 18.f;
  const float u0 = (gi * both + 2 * ge * one) * 16.5f, u1 = both * 64.f * ((gi + 2 * ge + warps - 1) / warps);
  const float s0 = 2 * gs * one * 16.5f, s1 = one * 64.f * ((2 * gs + warps - 1) / warps);
  return WO > 1 && (s0 > s1 ? s0 : s1) < (u0 > u1 ? u0 : u1);
}
__host__ __device__ inline bool flex_lane_pairs(int faces, int warps) {
  const int g = (2 * faces + 31) / 32;
  return g <= 4 && g <= warps;
}

template <int ND, int NF, int WO, int NT, bool VISC>
__global__ void __launch_bounds__(NT) flex_kernel(const DevParams P, const double* __restrict__ qin,
                                                  const double* __restrict__ qbase, double* __restrict__ qout,
                                                  const double dt, const int kind, const int tx, const int ty) {
  using Sh = FlexShape<ND, NF, WO>;
  using Q = Eqs<ND, NF>;
  using N = Num64;
  constexpr int S = Sh::S, H = Sh::H, NW = NT / 32;
  extern __shared__ __align__(16) double flex_smem[];
  double* const sq = flex_smem;
  double* const wx = sq + Sh::nq(tx, ty);          // left values, then right values
  double* const wy = wx + 2 * Sh::nwx(tx, ty);
  double* const cx = wy + 2 * Sh::nwy(tx, ty);     // [kNumCoef][tx + 2], then [kNumCoef][ty + 2]
  double* const cy = cx + (WO > 1 ? kNumCoef * (tx + 2) : 0);

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int nx = P.n[0], ny = P.n[1];
  const int x0 = blockIdx.x * tx, y0 = ND > 1 ? blockIdx.y * ty : 0;
  const int tw = min(tx, nx - x0), th = ND > 1 ? min(ty, ny - y0) : 1;  // the cells this tile owns
  const int LX = tw + 2 * H, LY = ND > 1 ? th + 2 * H : 1, LXY = LX * LY;
  const int NCX = tw + 2, NCY = ND > 1 ? th + 2 : 0;
  const int HY = ND > 1 ? H : 0;
  const N u0 = num64_unit(P.inv_d[0]);
  auto num = [&](double x) { return lift(x, u0); };
  // x values: position c = 0 .. tw+1 (cell x0-1+c) of row; y values: position c of column
  auto wxi = [&](int v, int row, int c) { return (v * th + row) * NCX + c; };
  auto wyi = [&](int v, int c, int col) { return (v * NCY + c) * tw + col; };
  double* const wxl = wx;
  double* const wxr = wx + S * th * NCX;
  double* const wyl = wy;
  double* const wyr = wy + S * NCY * tw;
  // row r of the flux of x face f (left of cell f), y face f
  auto fxv = [&](int r, int row, int f) -> double& {
    return r < S ? wxr[wxi(r, row, f)] : wxl[wxi(r - S, row, f + 1)];
  };
  auto fyv = [&](int r, int f, int col) -> double& {
    return r < S ? wyr[wyi(r, f, col)] : wyl[wyi(r - S, f + 1, col)];
  };

  // ---- load + BCs + cons -> prim -------------------------------------------
  if constexpr (WO > 1) {  // constant tables: before the wait
    for (int it = tid; it < kNumCoef * NCX; it += NT) {
      const int k = it / NCX, c = it - k * NCX;
      cx[it] = __ldg(P.coef[0] + k * P.cstride[0] + clamp_coef_index(x0 - 1 + c, nx) + P.coff);
    }
    if constexpr (ND > 1) {
      for (int it = tid; it < kNumCoef * NCY; it += NT) {
        const int k = it / NCY, c = it - k * NCY;
        cy[it] = __ldg(P.coef[1] + k * P.cstride[1] + clamp_coef_index(y0 - 1 + c, ny) + P.coff);
      }
    }
  }
  griddep_wait();  // the state below is the previous stage's output
  if (kind != kRkEuler && kind != kRhsOnly) {
    // the RK base register's lines of the tile, read only by the last phase
    const int lines = (tw * 8 + 127) / 128 + 1;
    for (int it = tid; it < S * th * lines; it += NT) {
      const int line = it % lines, r = it / lines, row = r % th, v = r / th;
      const int gx = min(x0 + line * 16, x0 + tw - 1);
      asm volatile("prefetch.global.L2 [%0];" ::"l"(qbase + (int64_t)(y0 + row) * P.sy + gx + v * P.sv));
    }
  }
  for (int c = tid; c < LXY; c += NT) {
    const int ly = c / LX, lx = c - ly * LX;
    // corners are never read, except the four diagonal neighbours of the
    // tile that the viscous cross derivatives use
    const bool hx = lx < H || lx >= H + tw, hy = ND > 1 && (ly < H || ly >= H + th);
    if (hx && hy && !(VISC && (lx == H - 1 || lx == H + tw) && (ly == H - 1 || ly == H + th))) continue;
    bool fx, fy;
    int64_t vs;
    const double* src = tile_cell<ND, H>(P, qin, x0 - H + lx, ND > 1 ? y0 - H + ly : 0, vs, fx, fy);
    double q[S];
#pragma unroll
    for (int v = 0; v < S; ++v) q[v] = __ldg(src + v * vs);
    if (fx) q[Q::MOM] = -q[Q::MOM];
    if (ND > 1 && fy) q[Q::MOM + 1] = -q[Q::MOM + 1];
    cons_to_prim<ND, NF>(q, P, u0);
#pragma unroll
    for (int v = 0; v < S; ++v) sq[v * LXY + c] = q[v];
  }
  __syncthreads();
  griddep_launch_dependents();

  // ---- WENO in every direction ------------------------------------------------
  // Groups of 32 items: the interior positions of x, of y (both face values),
  // then the positions just outside the tile, which feed one face each
  // (weno_cell_side, the same bits) -- first those that need the right value,
  // then those that need the left one.
  {
    const N eps = num(P.weno_eps);
    const int ni = S * th * tw, gi = (ni + 31) >> 5;
    const int nex = S * th, gex = (nex + 31) >> 5;
    const int ney = ND > 1 ? S * tw : 0, gey = (ney + 31) >> 5;
    const int gint = ND * gi, groups = gint + 2 * gex + 2 * gey;
    const int ns = S * (tw + 1), gs1 = (ns + 31) >> 5;
    const bool sides = ND == 1 && flex_sides<WO>(gi, gex, gs1, NW);
    // small 1-D tiles: every face value an item of its own, the right values
    // of cells -1 .. tw-1, then the left ones of cells 0 .. tw
    for (int g = sides ? warp : 2 * gs1; g < 2 * gs1; g += NW) {
      const bool left = g >= gs1;
      const int it = (left ? g - gs1 : g) * 32 + lane;
      if (it >= ns) continue;
      const int v = it / (tw + 1), c0 = it - v * (tw + 1), col = left ? c0 : c0 - 1;
      const double* at = sq + v * LXY + col + H;
      N s[5];
#pragma unroll
      for (int k = 0; k < 5; ++k) s[k] = num(k - 2 >= -(WO / 2) && k - 2 <= WO / 2 ? at[k - 2] : 0.0);
      // one code for both sides: the side's coefficients in the left's places
      double c[kCoefRec];
      if constexpr (WO > 1) {
#pragma unroll
        for (int k = 0; k < kNumCoef; ++k) {
          const int from = left ? k : k >= kPL && k < kPL + 6 ? k + (kPR - kPL) : k >= kDL && k < kDL + 3 ? k + (kDR - kDL) : k;
          c[k] = cx[from * NCX + col + 1];
        }
      }
      (left ? wxl : wxr)[wxi(v, 0, col + 1)] = low(weno_cell_side<WO, 0, N>(NumCoef<N>{c, u0}, s, eps));
    }
    for (int g = sides ? groups : warp; g < groups; g += NW) {
      if (g < gint) {
        const bool ydir = ND > 1 && g >= gi;
        const int it = (ydir ? g - gi : g) * 32 + lane;
        if (it >= ni) continue;
        const int r = it / tw, col = it - r * tw, v = r / th, row = r - v * th;
        const double* at = sq + v * LXY + (row + HY) * LX + col + H;
        const int st = ydir ? LX : 1;
        const double* cf = ydir ? cy + row + 1 : cx + col + 1;
        const int cs = ydir ? NCY : NCX;
        N s[5], vl, vr;
#pragma unroll
        for (int k = 0; k < 5; ++k) s[k] = num(k - 2 >= -(WO / 2) && k - 2 <= WO / 2 ? at[(k - 2) * st] : 0.0);
        double c[kCoefRec];
        if constexpr (WO > 1) {
#pragma unroll
          for (int k = 0; k < kNumCoef; ++k) c[k] = cf[k * cs];
        }
        weno_cell<WO, N>(NumCoef<N>{c, u0}, s, eps, vl, vr);
        if (ydir) {
          wyl[wyi(v, row + 1, col)] = low(vl);
          wyr[wyi(v, row + 1, col)] = low(vr);
        } else {
          wxl[wxi(v, row, col + 1)] = low(vl);
          wxr[wxi(v, row, col + 1)] = low(vr);
        }
      } else {
        int e = g - gint;
        const bool ydir = ND > 1 && e >= 2 * gex;
        if (ydir) e -= 2 * gex;
        const int gs = ydir ? gey : gex, n = ydir ? ney : nex;
        const bool left = e >= gs;  // the position after the tile: its left value
        const int it = (left ? e - gs : e) * 32 + lane;
        if (it >= n) continue;
        const int ext = ydir ? tw : th, v = it / ext, t = it - v * ext;
        // position 0 or tw + 1 (th + 1) of line t
        const int col = ydir ? t : (left ? tw : -1), row = ydir ? (left ? th : -1) : t;
        const double* at = sq + v * LXY + (row + HY) * LX + col + H;
        const int st = ydir ? LX : 1;
        const double* cf = ydir ? cy + row + 1 : cx + col + 1;
        const int cs = ydir ? NCY : NCX;
        N s[5];
#pragma unroll
        for (int k = 0; k < 5; ++k) s[k] = num(k - 2 >= -(WO / 2) && k - 2 <= WO / 2 ? at[(k - 2) * st] : 0.0);
        double c[kCoefRec];
        if constexpr (WO > 1) {
#pragma unroll
          for (int k = 0; k < kNumCoef; ++k) c[k] = cf[k * cs];
        }
        if (left) {
          const double w = low(weno_cell_side<WO, 0, N>(NumCoef<N>{c, u0}, s, eps));
          if (ydir) wyl[wyi(v, row + 1, col)] = w;
          else wxl[wxi(v, row, col + 1)] = w;
        } else {
          const double w = low(weno_cell_side<WO, 1, N>(NumCoef<N>{c, u0}, s, eps));
          if (ydir) wyr[wyi(v, row + 1, col)] = w;
          else wxr[wxi(v, row, col + 1)] = w;
        }
      }
    }
  }
  __syncthreads();

  // ---- HLLC in every direction ---------------------------------------------------
  {
    N gam_i[NF], pi_i[NF];
#pragma unroll
    for (int f = 0; f < NF; ++f) {
      gam_i[f] = num(P.gammas[f]);
      pi_i[f] = num(P.pi_infs[f]);
    }
    const int nfx = (tw + 1) * th, gx = (nfx + 31) >> 5;
    const int nfy = ND > 1 ? tw * (th + 1) : 0, gy = (nfy + 31) >> 5;
    auto U = [&](int c, int x, int y) { return num(sq[(Q::MOM + c) * LXY + y * LX + x]); };
    // few faces in 1-D: two lanes to a face, each with one of its states until
    // they meet
    const bool pairs = ND == 1 && !VISC && flex_lane_pairs(nfx, NW);
    if constexpr (ND == 1 && !VISC) {
      for (int g = warp; pairs && g < (2 * nfx + 31) >> 5; g += NW) {
        const int f0 = g * 16 + (lane >> 1), f = min(f0, tw);  // every lane of the warp takes part
        const bool mine = (lane & 1) != 0;                     // the right state
        const int gface = x0 - 1 + f;
        const bool lfr = gface == -1 && P.bc_beg[0] == -4, rfl = gface == nx - 1 && P.bc_end[0] == -4;
        N qL[S], qR[S], q[S], F[S], us;
#pragma unroll
        for (int v = 0; v < S; ++v) {
          const N a = num(wxr[wxi(v, 0, f)]), b = num(wxl[wxi(v, 0, f + 1)]);
          qL[v] = lfr ? b : a;
          qR[v] = rfl ? a : b;
          q[v] = mine ? qR[v] : qL[v];
        }
        const HllcSide<N> own = hllc_side<ND, NF, N>(q, gam_i, pi_i);
        const HllcSide<N> other{num(__shfl_xor_sync(0xffffffffu, low(own.rho), 1)),
                                num(__shfl_xor_sync(0xffffffffu, low(own.E), 1)),
                                num(__shfl_xor_sync(0xffffffffu, low(own.c), 1))};
        hllc_solve<ND, NF, 0, N>(qL, qR, mine ? other : own, mine ? own : other, F, us);
        __syncwarp();  // the face's states are read by both lanes
        if (f0 <= tw && !mine) {
#pragma unroll
          for (int v = 0; v < S; ++v) fxv(v, 0, f) = low(F[v]);
          fxv(S, 0, f) = low(us);
        }
      }
    }
    for (int g = pairs ? gx + gy : warp; g < gx + gy; g += NW) {
      N qL[S], qR[S], F[S], us;
      if (g < gx) {
        const int it = g * 32 + lane;
        if (it >= nfx) continue;
        const int row = it / (tw + 1), f = it - row * (tw + 1);
        const int gface = x0 - 1 + f;                              // face gface + 1/2
        const bool lfr = gface == -1 && P.bc_beg[0] == -4;         // qL(-1) = qR(0)
        const bool rfl = gface == nx - 1 && P.bc_end[0] == -4;     // qR(m+1) = qL(m)
#pragma unroll
        for (int v = 0; v < S; ++v) {
          const N a = num(wxr[wxi(v, row, f)]), b = num(wxl[wxi(v, row, f + 1)]);
          qL[v] = lfr ? b : a;
          qR[v] = rfl ? a : b;
        }
        if constexpr (VISC) {
          N vs[ND], dxv[2] = {num(0.0), num(0.0)}, dyv[2] = {num(0.0), num(0.0)}, vf[3];
          hllc_face<ND, NF, 0, N, true>(qL, qR, gam_i, pi_i, F, us, vs);
          const ViscParams& V = *P.visc;
          if (V.fg[0] != nullptr) {  // weno_Re_flux = T: the prepared face gradients
            const int64_t plane = (int64_t)(ND > 1 ? ny : 1) * (nx + 1);
            const double* gr = V.fg[0] + (int64_t)(y0 + row) * (nx + 1) + (gface + 1);
#pragma unroll
            for (int c = 0; c < ND; ++c) {
              dxv[c] = num(__ldg(gr + (c * ND) * plane));
              if constexpr (ND > 1) dyv[c] = num(__ldg(gr + (c * ND + 1) * plane));
            }
          } else {
            const int ly = row + HY, lx = f + H - 1;  // the face's left cell
            const auto Dx = divisor(__ldg(V.dcc[0] + x0 + f));
#pragma unroll
            for (int c = 0; c < ND; ++c) {
              const N d = div_rn(U(c, lx + 1, ly) - U(c, lx, ly), Dx);
              dxv[c] = num(0.5) * (d + d);
            }
            if constexpr (ND > 1) {
              const auto D0 = divisor(__ldg(V.dcc[1] + y0 + row)), D1 = divisor(__ldg(V.dcc[1] + y0 + row + 1));
#pragma unroll
              for (int c = 0; c < ND; ++c) {
                auto Ly = [&](int x) { return div_rn(U(c, x, ly) - U(c, x, ly - 1), D0); };
                auto Ry = [&](int x) { return div_rn(U(c, x, ly + 1) - U(c, x, ly), D1); };
                const N A = num(0.25) * (Ly(lx + 1) + Ry(lx + 1) + Ly(lx) + Ry(lx));
                dyv[c] = num(0.5) * (A + A);
              }
            }
          }
          viscous_face_flux<ND, NF, 0, N>(qL, qR, V, vs, dxv, dyv, vf);
#pragma unroll
          for (int t = 0; t < 3; ++t) fxv(S + 1 + t, row, f) = low(vf[t]);
        } else {
          hllc_face<ND, NF, 0, N>(qL, qR, gam_i, pi_i, F, us);
        }
#pragma unroll
        for (int v = 0; v < S; ++v) fxv(v, row, f) = low(F[v]);
        fxv(S, row, f) = low(us);
      } else if constexpr (ND > 1) {
        const int it = (g - gx) * 32 + lane;
        if (it >= nfy) continue;
        const int f = it / tw, col = it - f * tw;
        const int gface = y0 - 1 + f;
        const bool lfr = gface == -1 && P.bc_beg[1] == -4;
        const bool rfl = gface == ny - 1 && P.bc_end[1] == -4;
#pragma unroll
        for (int v = 0; v < S; ++v) {
          const N a = num(wyr[wyi(v, f, col)]), b = num(wyl[wyi(v, f + 1, col)]);
          qL[v] = lfr ? b : a;
          qR[v] = rfl ? a : b;
        }
        if constexpr (VISC) {
          N vs[ND], dxv[2], dyv[2], vf[3];
          hllc_face<ND, NF, 1, N, true>(qL, qR, gam_i, pi_i, F, us, vs);
          const ViscParams& V = *P.visc;
          if (V.fg[1] != nullptr) {
            const int64_t plane = (int64_t)(ny + 1) * nx;
            const double* gr = V.fg[1] + (int64_t)(gface + 1) * nx + x0 + col;
#pragma unroll
            for (int c = 0; c < 2; ++c) {
              dxv[c] = num(__ldg(gr + (c * 2) * plane));
              dyv[c] = num(__ldg(gr + (c * 2 + 1) * plane));
            }
          } else {
            const int ly = f + H - 1, lx = col + H;  // the face's lower cell
            const auto Dy = divisor(__ldg(V.dcc[1] + y0 + f));
            const auto D0 = divisor(__ldg(V.dcc[0] + x0 + col)), D1 = divisor(__ldg(V.dcc[0] + x0 + col + 1));
#pragma unroll
            for (int c = 0; c < 2; ++c) {
              auto Lx = [&](int y) { return div_rn(U(c, lx, y) - U(c, lx - 1, y), D0); };
              auto Rx = [&](int y) { return div_rn(U(c, lx + 1, y) - U(c, lx, y), D1); };
              const N A = num(0.25) * (Lx(ly + 1) + Rx(ly + 1) + Lx(ly) + Rx(ly));
              dxv[c] = num(0.5) * (A + A);
              const N d = div_rn(U(c, lx, ly + 1) - U(c, lx, ly), Dy);
              dyv[c] = num(0.5) * (d + d);
            }
          }
          viscous_face_flux<ND, NF, 1, N>(qL, qR, V, vs, dxv, dyv, vf);
#pragma unroll
          for (int t = 0; t < 3; ++t) fyv(S + 1 + t, f, col) = low(vf[t]);
        } else {
          hllc_face<ND, NF, 1, N>(qL, qR, gam_i, pi_i, F, us);
        }
#pragma unroll
        for (int v = 0; v < S; ++v) fyv(v, f, col) = low(F[v]);
        fyv(S, f, col) = low(us);
      }
    }
  }
  __syncthreads();

  // ---- flux divergence + RK: one (variable, cell) per thread ----------------------
  const int cells = tw * th;
  bool bad = false;
  auto finish = [&](auto kind_c) {
    constexpr int KIND = decltype(kind_c)::value;
    for (int it = tid; it < S * cells; it += NT) {
      const int v = it / cells, e = it - v * cells, row = e / tw, col = e - row * tw;
      const int64_t o = (int64_t)(y0 + row) * P.sy + (x0 + col) + v * P.sv;
      double b = 0.0, in = 0.0;
      if constexpr (KIND != kRhsOnly) {
        b = __ldg(qbase + o);
        in = KIND == kRkEuler ? b : __ldg(qin + o);
      }
      const N a = num(sq[v * LXY + (row + HY) * LX + col + H]);  // the volume fraction, for v >= ADV
      const N ix = num(__ldg(P.inv_d[0] + x0 + col));
      N r = ix * (num(fxv(v, row, col)) - num(fxv(v, row, col + 1)));
      if (v >= Q::ADV) r = mul_add(ix * a, num(fxv(S, row, col + 1)) - num(fxv(S, row, col)), r);
      // the viscous row of momentum d (d) and of the energy (2)
      const int vr = S + 1 + (v == Q::E ? 2 : v - Q::MOM);
      const bool vis = VISC && v >= Q::MOM && v <= Q::E;
      if (vis) r = mul_add(ix, num(fxv(vr, row, col)) - num(fxv(vr, row, col + 1)), r);  // m_rhs.fpp:591-603
      if constexpr (ND > 1) {
        const N iy = num(__ldg(P.inv_d[1] + y0 + row));
        r = mul_add(iy, num(fyv(v, row, col)) - num(fyv(v, row + 1, col)), r);
        if (v >= Q::ADV) r = mul_add(iy * a, num(fyv(S, row + 1, col)) - num(fyv(S, row, col)), r);
        if (vis) r = mul_add(iy, num(fyv(vr, row, col)) - num(fyv(vr, row + 1, col)), r);  // m_rhs.fpp:639-651
      }
      double out;
      if constexpr (KIND == kRhsOnly) out = low(r);
      else out = rk_combine(KIND, num(b), num(in), num(dt), r);
      bad |= not_finite(out);
      qout[o] = out;
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
  // state of the tile back, which this block stored
  if (P.monitor) {
    __syncthreads();
    bool nonphys = false;
    double icfl = 0.0;
    for (int e = tid; e < cells; e += NT) {
      const int row = e / tw, col = e - row * tw;
      const int64_t o = (int64_t)(y0 + row) * P.sy + (x0 + col);
      double qn[S], inv[ND];
#pragma unroll
      for (int v = 0; v < S; ++v) qn[v] = __ldcg(qout + o + v * P.sv);
      inv[0] = __ldg(P.inv_d[0] + x0 + col);
      if constexpr (ND > 1) inv[1] = __ldg(P.inv_d[1] + y0 + row);
      bool np;
      const double c = cell_icfl<ND, NF>(qn, P, dt, inv, np);
      nonphys |= np;
      if (!(c <= icfl)) icfl = c;  // keeps NaN
    }
    if (nonphys && P.status) atomicOr(P.status, MFC_FLAG_NEG_PRESSURE);
    monitor_max(P.monitor, icfl);
  }
  if (bad && P.status) atomicOr(P.status, MFC_FLAG_NAN);
}

// One directional sweep of a plain FP64 3-D stage (the work of sweep_kernel,
// mfc_sweep.cuh: the same work buffers, operations and order, hence the same
// bits) on tiles sized at run time: ta cells along the sweep for tb
// pencils side by side.  Bound by the FP64 unit like flex_kernel; what a fixed tile loses
// is the reconstructions beyond its two ends (18 positions for 16 cells, all
// formed two-sided) and the rounding of 97x80x71 cells to 32- and 16-cell
// tiles.  Tiles as long as the line where shared memory allows have two
// one-sided end positions per line instead.
//
// Shared memory follows the lanes: along the sweep for the x sweep, across
// the pencils (x fastest) for y and z, so that loads and stores of global
// memory are coalesced and shared-memory accesses free of conflicts.
//
// Measured (ms a step, before: the fastest fixed tile, sweep_kernel with 320
// threads): 48x40x33 1.39 -> 0.97, 97x80x71 9.14 -> 7.54, 200x60x90 15.5 ->
// 13.8, 128^3 26.05 -> 26.01, 256^3 204.4 -> 198.6.
template <int NF, int WO, int DIR>
struct FlexSweepShape {
  static constexpr int S = Eqs<3, NF>::S, H = (WO + 1) / 2;
  static size_t bytes(int ta, int np) {
    return sizeof(double) * ((size_t)S * np * (ta + 2 * H) + 2 * (size_t)S * np * (ta + 2) +
                             (WO > 1 ? (size_t)kNumCoef * (ta + 2) : 0));
  }
};

template <int NF, int WO, int NT, int DIR>
__global__ void __launch_bounds__(NT) flex_sweep_kernel(const DevParams P, const double* __restrict__ qin,
                                                        const double* __restrict__ qbase, double* __restrict__ qout,
                                                        const double dt, const int kind, const int ta, const int tb) {
  using Sh = FlexSweepShape<NF, WO, DIR>;
  using Q = Eqs<3, NF>;
  using N = Num64;
  constexpr int S = Sh::S, H = Sh::H, NW = NT / 32;
  constexpr int OA = DIR, OB = DIR == 0 ? 1 : 0, OC = DIR == 2 ? 1 : 2;  // axis index of a, b, c
  extern __shared__ __align__(16) double flex_smem[];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int na = P.n[OA], nb = P.n[OB];
  const int ia = blockIdx.x % ((na + ta - 1) / ta), ibc = blockIdx.x / ((na + ta - 1) / ta);
  const int nbt = (nb + tb - 1) / tb;
  const int a0 = ia * ta, b0 = (ibc % nbt) * tb, gc = ibc / nbt;
  const int ea = min(ta, na - a0), NP = min(tb, nb - b0);  // the cells along and the pencils of this tile
  const int LA = ea + 2 * H, NCA = ea + 2, NFA = ea + 1;
  double* const sq = flex_smem;                 // [S][pencil][LA], or [S][LA][pencil] for y and z
  double* const wl = sq + S * tb * (ta + 2 * H);
  double* const wr = wl + S * NP * NCA;
  double* const cf = wl + 2 * S * tb * (ta + 2);  // [kNumCoef][NCA]
  const N u0 = num64_unit(P.inv_d[0]);
  auto num = [&](double x) { return lift(x, u0); };
  const int sa = DIR == 0 ? 1 : NP;  // stride along the sweep
  auto qi = [&](int v, int p, int la) { return DIR == 0 ? (v * NP + p) * LA + la : (v * LA + la) * NP + p; };
  auto wi = [&](int v, int p, int c) { return DIR == 0 ? (v * NP + p) * NCA + c : (v * NCA + c) * NP + p; };
  // item it of e x NP (x S) items: position along the sweep, pencil, variable
  auto split = [&](int it, int e, int& a, int& p, int& v) {
    if (DIR == 0) {
      const int r = it / e;
      a = it - r * e;
      v = r / NP;
      p = r - v * NP;
    } else {
      const int r = it / NP;
      p = it - r * NP;
      v = r / e;
      a = r - v * e;
    }
  };
  // element offset of cell a of pencil p
  auto offset = [&](int a, int p) {
    int x, y, z;
    sweep_coords<DIR>(a0 + a, b0 + p, gc, x, y, z);
    return (int64_t)z * P.sz + (int64_t)y * P.sy + x;
  };
  // row r of the flux of face f (left of cell f) of pencil p, in place of the
  // two states it is solved from
  auto fv = [&](int r, int p, int f) -> double& { return r < S ? wr[wi(r, p, f)] : wl[wi(r - S, p, f + 1)]; };

  if constexpr (WO > 1) {  // constant tables: before the wait
    for (int it = tid; it < kNumCoef * NCA; it += NT) {
      const int k = it / NCA, c = it - k * NCA;
      cf[it] = __ldg(P.coef[DIR] + k * P.cstride[DIR] + clamp_coef_index(a0 - 1 + c, na) + P.coff);
    }
  }
  double* const rhs_buf = reinterpret_cast<double*>(P.work);
  // the primitives of the stage input: written by the x sweep, read by y and z
  double* const gprim = rhs_buf + (int64_t)S * P.sv;
  griddep_wait();
  if constexpr (DIR > 0) {
    // the last phase's operands, into L2: the partial RHS and, on the z
    // sweep, the RK registers
    const int arrays = DIR == 1 || kind == kRhsOnly ? 1 : (kind == kRkEuler ? 2 : 3);
    const int lines = (NP * 8 + 127) / 128 + 1, rows = S * ea;
    for (int it = tid; it < arrays * rows * lines; it += NT) {
      const int line = it % lines, r = it / lines, arr = r / rows, l = r - arr * rows;
      const int v = l % S, a = l / S;
      const int64_t o = offset(a, min(line * 16, NP - 1)) + v * P.sv;
      const double* ptr = arr == 0 ? rhs_buf + o : arr == 1 ? qbase + o : qin + o;
      asm volatile("prefetch.global.L2 [%0];" ::"l"(ptr));
    }
  }

  // ---- load + BCs (+ cons -> prim on the x sweep) -----------------------------
  const int64_t stride[3] = {1, P.sy, P.sz};
  for (int it = tid; it < NP * LA; it += NT) {
    int la, p, dummy_v;
    split(it, LA, la, p, dummy_v);
    const int gb = b0 + p;
    const int ra = a0 - H + la;
    bool fa = false;
    // processor boundary along the sweep: the neighbour's halo buffer
    const int side = ra < 0 ? (P.bc_beg[OA] >= 0 ? 0 : -1) : (ra >= na && P.bc_end[OA] >= 0 ? 1 : -1);
    const double* src;
    int64_t vs = P.sv, own = -1;
    if (side >= 0) {
      const int d = side == 0 ? -1 - ra : ra - na;
      int x, y, z;
      sweep_coords<DIR>(d, gb, gc, x, y, z);
      const int nx = P.n[0], ny = P.n[1], nz = P.n[2];
      const double* h = P.halo[2 * DIR + side];
      if (DIR == 0) { src = h + ((int64_t)z * ny + y) * H + d; vs = (int64_t)nz * ny * H; }
      else if (DIR == 1) { src = h + ((int64_t)z * H + d) * nx + x; vs = (int64_t)nz * H * nx; }
      else { src = h + ((int64_t)d * ny + y) * nx + x; vs = (int64_t)H * ny * nx; }
    } else {
      const int ga = map_cell(ra, na, P.bc_beg[OA], P.bc_end[OA], &fa);
      const int64_t o = ga * stride[OA] + gb * stride[OB] + gc * stride[OC];
      if constexpr (DIR > 0) {
        // the stored primitives; a reflected cell's normal velocity negated
#pragma unroll
        for (int v = 0; v < S; ++v) {
          const double w = __ldg(gprim + o + v * P.sv);
          sq[qi(v, p, la)] = (fa && v == Q::MOM + DIR) ? -w : w;
        }
        continue;
      }
      src = qin + o;
      if (la >= H && la < H + ea) own = o;
    }
    double q[S];
#pragma unroll
    for (int v = 0; v < S; ++v) q[v] = __ldg(src + v * vs);
    if (fa) q[Q::MOM + DIR] = -q[Q::MOM + DIR];
    cons_to_prim<3, NF>(q, P, u0);
#pragma unroll
    for (int v = 0; v < S; ++v) sq[qi(v, p, la)] = q[v];
    if (DIR == 0 && own >= 0) {
#pragma unroll
      for (int v = 0; v < S; ++v) gprim[own + v * P.sv] = q[v];
    }
  }
  __syncthreads();
  griddep_launch_dependents();

  // ---- WENO: interior positions, then the two end positions of every line -----
  {
    const N eps = num(P.weno_eps);
    const int ni = S * NP * ea, gi = (ni + 31) >> 5, ne = S * NP, ge = (ne + 31) >> 5;
    for (int g = warp; g < gi + 2 * ge; g += NW) {
      const bool end = g >= gi, left = g >= gi + ge;  // left: the position after the tile, its left value
      const int it = (end ? (left ? g - gi - ge : g - gi) : g) * 32 + lane;
      if (it >= (end ? ne : ni)) continue;
      int a, p, v;
      split(it, end ? 1 : ea, a, p, v);
      if (end) a = left ? ea : -1;
      const double* at = sq + qi(v, p, a + H);
      N s[5];
#pragma unroll
      for (int k = 0; k < 5; ++k) s[k] = num(k - 2 >= -(WO / 2) && k - 2 <= WO / 2 ? at[(k - 2) * sa] : 0.0);
      double c[kCoefRec];
      if constexpr (WO > 1) {
#pragma unroll
        for (int k = 0; k < kNumCoef; ++k) c[k] = cf[k * NCA + a + 1];
      }
      if (!end) {
        N vl, vr;
        weno_cell<WO, N>(NumCoef<N>{c, u0}, s, eps, vl, vr);
        wl[wi(v, p, a + 1)] = low(vl);
        wr[wi(v, p, a + 1)] = low(vr);
      } else if (left) {
        wl[wi(v, p, a + 1)] = low(weno_cell_side<WO, 0, N>(NumCoef<N>{c, u0}, s, eps));
      } else {
        wr[wi(v, p, a + 1)] = low(weno_cell_side<WO, 1, N>(NumCoef<N>{c, u0}, s, eps));
      }
    }
  }
  __syncthreads();

  // ---- HLLC -------------------------------------------------------------------------
  {
    N gam_i[NF], pi_i[NF];
#pragma unroll
    for (int f = 0; f < NF; ++f) {
      gam_i[f] = num(P.gammas[f]);
      pi_i[f] = num(P.pi_infs[f]);
    }
    for (int it = tid; it < NP * NFA; it += NT) {
      int f, p, dummy_v;
      split(it, NFA, f, p, dummy_v);
      const int gface = a0 - 1 + f;
      const bool lfr = gface == -1 && P.bc_beg[OA] == -4, rfl = gface == na - 1 && P.bc_end[OA] == -4;
      N qL[S], qR[S], F[S], us;
#pragma unroll
      for (int v = 0; v < S; ++v) {
        const N l = num(wr[wi(v, p, f)]), r = num(wl[wi(v, p, f + 1)]);
        qL[v] = lfr ? r : l;
        qR[v] = rfl ? l : r;
      }
      hllc_face<3, NF, DIR, N>(qL, qR, gam_i, pi_i, F, us);
#pragma unroll
      for (int v = 0; v < S; ++v) fv(v, p, f) = low(F[v]);
      fv(S, p, f) = low(us);
    }
  }
  __syncthreads();

  // ---- divergence, accumulation, RK on the last sweep: one (variable, cell) per thread
  const int cells = NP * ea;
  bool bad = false;
  auto finish = [&](auto kind_c) {
    constexpr int KIND = decltype(kind_c)::value;
    for (int it = tid; it < S * cells; it += NT) {
      int a, p, v;
      split(it, ea, a, p, v);
      const int64_t o = offset(a, p) + v * P.sv;
      double part = 0.0, b = 0.0, in = 0.0;
      if constexpr (DIR > 0) part = rhs_buf[o];
      if constexpr (DIR == 2 && KIND != kRhsOnly) {
        b = __ldg(qbase + o);
        in = KIND == kRkEuler ? b : __ldg(qin + o);
      }
      const N inv = num(__ldg(P.inv_d[DIR] + a0 + a));
      const N diff = num(fv(v, p, a)) - num(fv(v, p, a + 1));
      N r = DIR == 0 ? inv * diff : mul_add(inv, diff, num(part));
      if (v >= Q::ADV) r = mul_add(inv * num(sq[qi(v, p, a + H)]), num(fv(S, p, a + 1)) - num(fv(S, p, a)), r);
      if constexpr (DIR < 2) {
        rhs_buf[o] = low(r);
      } else {
        double out;
        if constexpr (KIND == kRhsOnly) out = low(r);
        else out = rk_combine(KIND, num(b), num(in), num(dt), r);
        bad |= not_finite(out);
        qout[o] = out;
      }
    }
  };
  if constexpr (DIR < 2) {
    finish(KindC<kRhsOnly>{});
  } else {
    switch (kind) {
      case kRkEuler: finish(KindC<kRkEuler>{}); break;
      case kRk2Final: finish(KindC<kRk2Final>{}); break;
      case kRk3Mid: finish(KindC<kRk3Mid>{}); break;
      case kRk3Final: finish(KindC<kRk3Final>{}); break;
      default: finish(KindC<kRhsOnly>{}); break;
    }
    if (P.monitor) {  // the new state of the tile, which this block stored
      __syncthreads();
      bool nonphys = false;
      double icfl = 0.0;
      for (int it = tid; it < cells; it += NT) {
        int a, p, dummy_v;
        split(it, ea, a, p, dummy_v);
        const int64_t o = offset(a, p);
        double qn[S];
#pragma unroll
        for (int v = 0; v < S; ++v) qn[v] = __ldcg(qout + o + v * P.sv);
        const double inv[3] = {__ldg(P.inv_d[0] + b0 + p), __ldg(P.inv_d[1] + gc), __ldg(P.inv_d[2] + a0 + a)};
        bool np;
        const double c = cell_icfl<3, NF>(qn, P, dt, inv, np);
        nonphys |= np;
        if (!(c <= icfl)) icfl = c;  // keeps NaN
      }
      if (nonphys && P.status) atomicOr(P.status, MFC_FLAG_NEG_PRESSURE);
      monitor_max(P.monitor, icfl);
    }
    if (bad && P.status) atomicOr(P.status, MFC_FLAG_NAN);
  }
}

}  // namespace mfc
