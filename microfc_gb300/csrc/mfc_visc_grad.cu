// weno_Re_flux = T: the velocity gradients of the viscous stresses from
// WENO reconstructions instead of finite differences.  The reference
// (m_viscous.fpp:176-216, 381-591; m_rhs.fpp:512-528; the averaging in
// s_compute_viscous_source_flux, m_riemann_solvers.fpp:683-902):
//
//   1. every velocity component u_c is WENO-reconstructed along each
//      direction d, and the cell-average gradient follows from the scalar
//      divergence theorem, G_cd = (1/ds) (u_c(right face) - u_c(left face));
//   2. every G_cd is WENO-reconstructed along the sweep direction, and the
//      face value is the mean of the right-face value of the cell before the
//      face and the left-face value of the cell after it.
//
// Kernels per RK stage prepare those face values from the stage input; the
// stage kernel's viscous flux reads them (ViscParams::fg).  The velocities
// are FP64 in every precision; the two reconstructions run in RT: FP64 for
// the plain path (the arithmetic and operation order of the oracle, so the
// result is bit-identical to it), FP32 for the split and gated paths, whose
// stage kernels take the gradients in FP32 anyway.  The buffers stay FP64
// (an FP32 value widened, so the stage kernel narrows it back exactly), but in
// 2-D the split and gated paths take one tiled kernel and FP32 pairs (below).
// Cells outside the domain take the boundary conditions by index mapping,
// as everywhere else.
//
// Regions (x0 = 0 .. nx-1, y0 = 0 .. ny-1 the interior):
//   x faces i+1/2, i = -1 .. nx-1, rows y0: need G on x = -3 .. nx+2, rows y0,
//     whose WENO along x reads u on x = -5 .. nx+4 and, for G_c1, along y on
//     rows -2 .. ny+1 (corner ghost cells);
//   y faces j+1/2, j = -1 .. ny-1, columns x0: need G on y = -3 .. ny+2,
//     columns x0.
// One launch computes G on the box x, y = -3 .. n+2 that holds both (each
// interior cell once; the 36 corner cells of the box are computed and not
// read), from the velocities of x, y = -5 .. n+4.
#include <cuda_runtime.h>

#include <algorithm>

#include "../../include/mfc_gpu.h"
#include "mfc_launch.h"

namespace mfc {
namespace {

// Velocity component c of cell (i, j) of state q, with the boundary
// conditions (the reflected normal component negated), as cons_to_prim
// computes it.
template <int ND, int NF>
__device__ __forceinline__ double velocity(const DevParams& P, const double* __restrict__ q, int c, int i, int j) {
  bool fx = false, fy = false;
  const int gx = map_cell(i, P.n[0], P.bc_beg[0], P.bc_end[0], &fx);
  const int gy = ND > 1 ? map_cell(j, P.n[1], P.bc_beg[1], P.bc_end[1], &fy) : 0;
  const int64_t o = (int64_t)gy * P.sy + gx;
  double rho = 0.0;
#pragma unroll
  for (int f = 0; f < NF; ++f) rho = rho + __ldg(q + o + f * P.sv);
  rho = fmax(rho, 1e-16);
  double m = __ldg(q + o + (NF + c) * P.sv);
  if ((c == 0 && fx) || (c == 1 && fy)) m = -m;
  return div_rn(m, divisor(rho));
}

// The velocities of the cells x = -5 .. nx+4 (and y = -5 .. ny+4 in 2-D)
// once, into vel[c][row][col] (row = y + 5, col = x + 5), which every
// stencil of the cell gradients reads.
template <int ND, int NF>
__global__ void __launch_bounds__(256) visc_velocities(const DevParams P, const double* __restrict__ q,
                                                      const int ncol, const int nrow, double* __restrict__ vel) {
  const int64_t cells = (int64_t)ncol * nrow;
  for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < cells; t += (int64_t)gridDim.x * blockDim.x) {
    const int col = (int)(t % ncol), row = (int)(t / ncol);
    const int i = col - 5, j = ND > 1 ? row - 5 : 0;
#pragma unroll
    for (int c = 0; c < ND; ++c) vel[(int64_t)c * cells + t] = velocity<ND, NF>(P, q, c, i, j);
  }
}

// The WENO coefficients of cell `cell` along direction d: FP64 from the
// context's grid tables, FP32 from the preparation's own table cft of that
// direction ([kNumCoef][n + 2 kCoefPad], then the inverse cell widths).
template <class RT>
__device__ __forceinline__ void coef_of(const DevParams& P, const float* __restrict__ cft, int d, int cell,
                                        RT (&c)[kCoefRec]) {
  const int gi = clamp_coef_index(cell, P.n[d]) + kCoefPad;
  if constexpr (sizeof(RT) == 4) {
    const int stride = P.n[d] + 2 * kCoefPad;
#pragma unroll
    for (int k = 0; k < kNumCoef; ++k) c[k] = __ldg(cft + k * stride + gi);
  } else {
#pragma unroll
    for (int k = 0; k < kNumCoef; ++k) c[k] = __ldg(P.coef[d] + k * P.cstride[d] + gi);
  }
}

// 1/ds of cell `cell` along direction d (w: the FP64 widths of the
// direction, cft: its FP32 table).
template <class RT>
__device__ __forceinline__ RT inverse_width(const DevParams& P, const double* __restrict__ w,
                                            const float* __restrict__ cft, int d, int cell) {
  const int gi = clamp_coef_index(cell, P.n[d]) + kCoefPad;
  if constexpr (sizeof(RT) == 4) return __ldg(cft + kNumCoef * (P.n[d] + 2 * kCoefPad) + gi);
  else return div_rn(1.0, divisor(__ldg(w + gi)));
}

// weno_cell on a record of RT coefficients, in the number type N.
template <class RT, class N>
__device__ __forceinline__ void grad_cell(const RT (&c)[kCoefRec], const N (&v)[5], const N& eps, const N& u0, N& vl,
                                          N& vr) {
  if constexpr (sizeof(RT) == 8) weno_cell<5, N>(NumCoef<N>{c, u0}, v, eps, vl, vr);
  else weno_cell<5, N>(c, v, eps, vl, vr);
}

// Step 1 on the ncol x nrow cells from (ib, jb): out[c*ND+d][row][col].
// B.w[d]: the cell widths ds of direction d for cells -kCoefPad ..
// n-1+kCoefPad; B.cf[d]: the FP32 table of the direction.
template <int ND, class RT>
__global__ void __launch_bounds__(256) visc_cell_gradients(const DevParams P, const ViscGradBuffers B,
                                                          const int vcol, const int vrow, const int ib, const int jb,
                                                          const int ncol, const int nrow, double* __restrict__ out) {
  const double* __restrict__ vel = B.vel;
  const int64_t cells = (int64_t)ncol * nrow;
  const int64_t vplane = (int64_t)vcol * vrow;
  using N = std::conditional_t<sizeof(RT) == 8, Num64, RT>;
  N u0;
  if constexpr (sizeof(RT) == 8) u0 = num64_unit(P.inv_d[0]);
  else u0 = RT(0);
  const N eps = lift(narrow<RT>(P.weno_eps), u0);
  for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < cells; t += (int64_t)gridDim.x * blockDim.x) {
    const int col = (int)(t % ncol), row = (int)(t / ncol);
    const int i = ib + col, j = jb + row;
#pragma unroll
    for (int d = 0; d < ND; ++d) {
      const int cell = d == 0 ? i : j;
      RT cf[kCoefRec];
      coef_of(P, B.cf[d], d, cell, cf);
      const RT inv = inverse_width<RT>(P, B.w[d], B.cf[d], d, cell);
#pragma unroll
      for (int c = 0; c < ND; ++c) {
        N st[5];
#pragma unroll
        for (int o = 0; o < 5; ++o) {
          const int vi = i + (d == 0 ? o - 2 : 0) + 5, vj = ND > 1 ? j + (d == 1 ? o - 2 : 0) + 5 : 0;
          st[o] = lift(narrow<RT>(__ldg(vel + c * vplane + (int64_t)vj * vcol + vi)), u0);
        }
        N vl, vr;
        grad_cell(cf, st, eps, u0, vl, vr);
        out[((int64_t)(c * ND + d) * nrow + row) * ncol + col] = widen(low(lift(inv, u0) * (vr - vl)));
      }
    }
  }
}

// Step 2: the face values, from the cell gradients G of the region
// ([c*ND+d][grow][gcol], origin (gib, gjb)).  Each cell's gradients are
// WENO-reconstructed once, both face values together (weno_cell: the same
// operations as the one-sided form, so the same bits), and face F (between
// cells F-1 and F, F = 0 .. n_dir) takes 0.5 (right value of cell F-1 + left
// value of cell F).  out[c*ND+d][...], the face index F along dir.
//
// x faces: a warp covers 31 faces of one row.  Lane L reconstructs cell
// base + L - 1 (clamped to the last cell needed, nx); lanes 1..31 write face
// base + L - 1 with the right value of lane L-1 (shuffle) and their own left
// value.  Every lane of a warp runs the same iterations (the loop bound is
// per warp), so the full-mask shuffles are safe.
template <int ND, class RT>
__global__ void __launch_bounds__(256) visc_face_gradients_x(const DevParams P, const float* __restrict__ cft,
                                                            const double* __restrict__ G, const int gib,
                                                            const int gjb, const int gncol, const int gnrow,
                                                            double* __restrict__ out) {
  const int nx = P.n[0], nf = nx + 1;
  const int nl = ND > 1 ? P.n[1] : 1;  // rows
  const int chunks = (nf + 30) / 31;
  const int64_t warps = (int64_t)chunks * nl;
  const int64_t plane_out = (int64_t)nf * nl;
  const int lane = threadIdx.x & 31;
  using N = std::conditional_t<sizeof(RT) == 8, Num64, RT>;
  N u0;
  if constexpr (sizeof(RT) == 8) u0 = num64_unit(P.inv_d[0]);
  else u0 = RT(0);
  const N eps = lift(narrow<RT>(P.weno_eps), u0);
  const int64_t stride = ((int64_t)gridDim.x * blockDim.x) >> 5;
  for (int64_t w = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5; w < warps; w += stride) {
    const int l = (int)(w / chunks), base = (int)(w % chunks) * 31;
    const int F = base + lane - 1;   // this lane's face (written by lanes 1..31 while F < nf)
    const int cell = min(F, nx);     // and its cell, -1 .. nx
    RT cf[kCoefRec];
    coef_of(P, cft, 0, cell, cf);
    const double* row = G + (int64_t)(l - gjb) * gncol + (cell - gib);
#pragma unroll
    for (int k = 0; k < ND * ND; ++k) {
      N st[5];
#pragma unroll
      for (int o = 0; o < 5; ++o) st[o] = lift(narrow<RT>(__ldg(row + (int64_t)k * gnrow * gncol + (o - 2))), u0);
      N vl, vr;
      grad_cell(cf, st, eps, u0, vl, vr);
      const RT right = __shfl_up_sync(0xffffffffu, low(vr), 1);  // face value of the cell before
      if (lane >= 1 && F < nf) out[k * plane_out + (int64_t)l * nf + F] = widen(low(lift(RT(0.5), u0) * (lift(right, u0) + vl)));
    }
  }
}

// y faces (2-D, FP64): a thread walks one column through a run of R faces (cells
// f0-1 .. f0+R-1), carrying each cell's right values to the next face.
template <int R>
__global__ void __launch_bounds__(256) visc_face_gradients_y(const DevParams P, const double* __restrict__ G,
                                                            const int gib, const int gjb, const int gncol,
                                                            const int gnrow, double* __restrict__ out) {
  const int nx = P.n[0], ny = P.n[1], nf = ny + 1;
  const int runs = (nf + R - 1) / R;
  const int64_t items = (int64_t)nx * runs;
  const int64_t plane_out = (int64_t)nf * nx;
  using N = Num64;
  const N u0 = num64_unit(P.inv_d[0]), eps = lift(P.weno_eps, u0);
  for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < items; t += (int64_t)gridDim.x * blockDim.x) {
    const int l = (int)(t % nx), f0 = (int)(t / nx) * R;
    N prev[4];
#pragma unroll 1
    for (int j = -1; j < R; ++j) {
      const int cell = f0 + j;  // -1 .. ny
      if (cell > ny) break;
      double cf[kCoefRec];
      coef_of(P, nullptr, 1, cell, cf);
      const double* col = G + (int64_t)(cell - gjb) * gncol + (l - gib);
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        N st[5];
#pragma unroll
        for (int o = 0; o < 5; ++o) st[o] = lift(__ldg(col + ((int64_t)k * gnrow + (o - 2)) * gncol), u0);
        N vl, vr;
        grad_cell(cf, st, eps, u0, vl, vr);
        if (j >= 0) out[k * plane_out + (int64_t)cell * nx + l] = low(lift(0.5, u0) * (prev[k] + vl));
        prev[k] = vr;
      }
    }
  }
}

// ---------------------------------------------------------------------------
// 2-D split and gated contexts: one tiled kernel in place of the cell- and
// face-gradient kernels, on pairs (d u/d x_d, d v/d x_d).
//
// The unfused FP32 kernels were bound by issue: 12 scalar reconstructions a
// cell with 12 IEEE divisions each, 27 coefficient loads per cell and
// direction, intermediates widened to FP64 through L2 (130 us a stage at
// 1024x512).  Here a block takes 32x16 faces of each direction: velocities
// with a halo of 5, both cell gradients with a halo of 3 and the face values
// live in shared memory, both components are reconstructed by packed FP32
// operations that round as weno_cell's do, and a uniform grid's coefficients
// come from the parameters.  Measured at 1024x512: 130 -> 49 us a stage with
// the velocities; a split weno_Re_flux step 604 -> 343 us.  Bound by FP32 issue.
constexpr int kGX = 32, kGY = 16, kGT = 256;
struct GradShape {
  static constexpr int UX = kGX + 9, UY = kGY + 9;    // velocities: x0-5 .. x0+kGX+3
  static constexpr int GX = kGX + 5, GY = kGY + 5;    // cell gradients: x0-3 .. x0+kGX+1
  static constexpr int PX = kGX + 1, PY = kGY + 1;    // reconstructed cells: x0-1 .. x0+kGX-1
  static constexpr int NU = UX * UY, NG = GX * GY, NX = PX * kGY, NY = PY * kGX;
  static constexpr size_t kBytes = sizeof(f32x2) * size_t(NU + 2 * NG + 4 * (NX > NY ? NX : NY));
};

// One pair's reconstruction from its stencil: weno_cell's operations in their
// order, rounded one by one, two variables at a time.  The quotients are
// Markstein's (Handbook of Floating-Point Arithmetic, 2nd ed., ch. 4.7): the
// reciprocal refined by a Newton step, the quotient corrected by its exact
// remainder -- the IEEE quotient but for rare last bits, at a third of its
// instructions, and the reciprocal of b_k^2 serves both faces, that of the
// sum all three weights.  A product that a sum takes is fma(a, b, nz) with
// nz = -0 in a register: ptxas contracts packed multiplies and adds whatever
// their rounding modifiers say.
//
// The weights do not change when all b_k are scaled alike, so each lane's are
// scaled by the power of two that brings its least b_k to [1, 2): b_k^2 of a
// uniform velocity (weno_eps^2) stays a normal number for every weno_eps that
// FP32 holds, and that of the smoothest stencil never overflows.  A stencil
// 2^63 times rougher has no weight either way; its b_k is cut there, which
// keeps the divisors inside the reciprocal's range (the Newton step of an
// infinity or a zero is not a number).  The scale and the cut cost 1 % of a
// step (340 -> 343 us at 1024x512) and change no bit of ordinary values.
__device__ __forceinline__ f32x2 f2_neg(f32x2 a) { return a ^ 0x8000000080000000ull; }
__device__ __forceinline__ f32x2 f2_reciprocal(f32x2 a) {
  const f32x2 r = f2_rcp(a);
  return f2_fma(r, f2_fma(f2_neg(a), r, f2_pack(1.f, 1.f)), r);
}
__device__ __forceinline__ f32x2 f2_quotient(f32x2 n, f32x2 d, f32x2 r) {
  const f32x2 q = f2_mul(n, r);
  return f2_fma(f2_fma(f2_neg(d), q, n), r, q);
}
// 2^-e of each lane, e the exponent of the lane's least value.
__device__ __forceinline__ f32x2 f2_scale_to_one(f32x2 a, f32x2 b, f32x2 c) {
  float a0, a1, b0, b1, c0, c1;
  f2_unpack(a, a0, a1);
  f2_unpack(b, b0, b1);
  f2_unpack(c, c0, c1);
  auto inverse = [](float x) { return __uint_as_float(0x7f000000u - (__float_as_uint(x) & 0x7f800000u)); };
  return f2_pack(inverse(fminf(fminf(a0, b0), c0)), inverse(fminf(fminf(a1, b1), c1)));
}
// The smaller of each lane and 2^63; NaN stays NaN.
__device__ __forceinline__ f32x2 f2_cut(f32x2 a) {
  float x, y;
  f2_unpack(a, x, y);
  asm("min.NaN.f32 %0, %0, 0f5F000000;" : "+f"(x));
  asm("min.NaN.f32 %0, %0, 0f5F000000;" : "+f"(y));
  return f2_pack(x, y);
}
template <class Coef>
__device__ __forceinline__ void grad_weno(const Coef& C, const f32x2 (&v)[5], const f32x2 eps, const f32x2 nz,
                                          f32x2& vL, f32x2& vR) {
  const f32x2 d1 = f2_sub(v[4], v[3]), d0 = f2_sub(v[3], v[2]), dm1 = f2_sub(v[2], v[1]), dm2 = f2_sub(v[1], v[0]);
  auto indicator = [&](const int k, const f32x2 a, const f32x2 b) {  // b_k
    const f32x2 t0 = f2_fma(f2_mul(C(kBeta + 3 * k), a), a, nz), t1 = f2_fma(f2_mul(C(kBeta + 3 * k + 1), a), b, nz),
                t2 = f2_fma(f2_mul(C(kBeta + 3 * k + 2), b), b, nz);
    return f2_add(f2_add(f2_add(t0, t1), t2), eps);
  };
  const f32x2 b0 = indicator(0, d1, d0), b1 = indicator(1, d0, dm1), b2 = indicator(2, dm1, dm2);
  const f32x2 scale = f2_scale_to_one(b0, b1, b2);
  auto square = [&](const f32x2 b) {
    const f32x2 t = f2_cut(f2_mul(b, scale));
    return f2_mul(t, t);
  };
  const f32x2 D0 = square(b0), D1 = square(b1), D2 = square(b2);
  const f32x2 r0 = f2_reciprocal(D0), r1 = f2_reciprocal(D1), r2 = f2_reciprocal(D2);
#pragma unroll
  for (int side = 0; side < 2; ++side) {
    const int kP = side ? kPR : kPL, kD = side ? kDR : kDL;
    const f32x2 p0 = f2_add(f2_add(v[2], f2_fma(C(kP + 0), d1, nz)), f2_fma(C(kP + 1), d0, nz));
    const f32x2 p1 = f2_add(f2_add(v[2], f2_fma(C(kP + 2), d0, nz)), f2_fma(C(kP + 3), dm1, nz));
    const f32x2 p2 = f2_add(f2_add(v[2], f2_fma(C(kP + 4), dm1, nz)), f2_fma(C(kP + 5), dm2, nz));
    const f32x2 a0 = f2_quotient(C(kD + 0), D0, r0), a1 = f2_quotient(C(kD + 1), D1, r1),
                a2 = f2_quotient(C(kD + 2), D2, r2);
    const f32x2 s = f2_add(f2_add(a0, a1), a2), rs = f2_reciprocal(s);
    const f32x2 val = f2_add(f2_add(f2_fma(f2_quotient(a0, s, rs), p0, nz), f2_fma(f2_quotient(a1, s, rs), p1, nz)),
                             f2_fma(f2_quotient(a2, s, rs), p2, nz));
    if (side) vR = val;
    else vL = val;
  }
}

// vel: the velocities as (u, v) pairs, [ny + 10][nx + 10] from x = y = -5.
// fx, fy: the face gradients, pairs of components: [d][ny][nx + 1] and
// [d][ny + 1][nx] (face F between cells F - 1 and F).
// UNI: the shared coefficients U of a uniform grid, else per-cell ones (two
// kernels: together their code missed the instruction cache).
template <bool UNI>
__global__ void __launch_bounds__(kGT) visc_gradients_tiled(const DevParams P, const __grid_constant__ GradCoef U,
                                                           const float* __restrict__ cfx,
                                                           const float* __restrict__ cfy,
                                                           const f32x2* __restrict__ vel, f32x2* __restrict__ fx,
                                                           f32x2* __restrict__ fy) {
  using Sh = GradShape;
  extern __shared__ __align__(16) f32x2 grad_smem[];
  f32x2* const su = grad_smem;          // [UY][UX]
  f32x2* const sg = su + Sh::NU;        // [d][GY][GX]
  f32x2* const sl = sg + 2 * Sh::NG;    // [d][..] left values
  f32x2* const sr = sl + 2 * (Sh::NX > Sh::NY ? Sh::NX : Sh::NY);
  const int tid = threadIdx.x, nx = P.n[0], ny = P.n[1];
  const unsigned tiles_x = nx / kGX + 1;
  const int x0 = blockIdx.x % tiles_x * kGX, y0 = blockIdx.x / tiles_x * kGY;
  const float eps = d2f_bits(P.weno_eps);  // cut like every value, where weno_eps_f is rounded
  const f32x2 eps2 = f2_pack(eps, eps);
  const f32x2 half = f2_pack(0.5f, 0.5f);
  // -0 in both lanes, opaque to the compiler as fma64_unit's constants are
  const uint32_t sign = 0x80000000u | (uint32_t)(__double2hiint(__ldg(P.inv_d[0])) >> 31);
  const f32x2 nz = (f32x2)sign << 32 | sign;
  griddep_wait();
  for (int it = tid; it < Sh::NU; it += kGT) {
    const int r = it / Sh::UX, c = it - r * Sh::UX;
    // cells past the buffer (partial tiles) are never used
    su[it] = __ldg(vel + (int64_t)min(y0 + r, ny + 9) * (nx + 10) + min(x0 + c, nx + 9));
  }
  __syncthreads();
  // with the coefficients of cell `cell` along direction d
  auto with_coef = [&](auto dir, const int cell, auto&& use) {
    constexpr int D = decltype(dir)::value;
    if constexpr (UNI) {
      use([&](int k) { return f32x2(U.rec[D][k]); }, f32x2(U.rec[D][kNumCoef]));
    } else {
      float c[kCoefRec];
      const float* cf = D == 0 ? cfx : cfy;
      coef_of<float>(P, cf, D, cell, c);
      const float inv = inverse_width<float>(P, nullptr, cf, D, cell);
      use([&](int k) { return f2_pack(c[k], c[k]); }, f2_pack(inv, inv));
    }
  };
  // step 1: the cell gradients that a face of the tile needs: the tile's rows
  // with all columns, then the other rows of the tile's columns
  constexpr int kA = kGY * Sh::GX, kB = (Sh::GY - kGY) * kGX;
  for (int it = tid; it < 2 * (kA + kB); it += kGT) {
    const int d = it >= kA + kB, i = d ? it - (kA + kB) : it;
    int gx, gy;
    if (i < kA) {
      gy = 3 + i / Sh::GX;
      gx = i % Sh::GX;
    } else {
      const int r = (i - kA) / kGX;
      gy = r < 3 ? r : kGY + r;
      gx = 3 + (i - kA) % kGX;
    }
    const f32x2* at = su + (gy + 2) * Sh::UX + gx + 2;  // the cell: x0 - 3 + gx
    f32x2 v[5], vl, vr;
    auto recon = [&](const auto& C, const f32x2 inv) {
      grad_weno(C, v, eps2, nz, vl, vr);
      sg[d * Sh::NG + gy * Sh::GX + gx] = f2_mul(inv, f2_sub(vr, vl));
    };
    if (d == 0) {
#pragma unroll
      for (int k = 0; k < 5; ++k) v[k] = at[k - 2];
      with_coef(KindC<0>{}, min(x0 - 3 + gx, nx + 2), recon);
    } else {
#pragma unroll
      for (int k = 0; k < 5; ++k) v[k] = at[(k - 2) * Sh::UX];
      with_coef(KindC<1>{}, min(y0 - 3 + gy, ny + 2), recon);
    }
  }
  __syncthreads();
  // step 2, x faces: both gradient pairs along the rows
  for (int it = tid; it < 2 * Sh::NX; it += kGT) {
    const int d = it >= Sh::NX, i = d ? it - Sh::NX : it, r = i / Sh::PX, c = i - r * Sh::PX;  // cell x0 - 1 + c
    const f32x2* at = sg + d * Sh::NG + (r + 3) * Sh::GX + c + 2;
    f32x2 v[5], vl, vr;
#pragma unroll
    for (int k = 0; k < 5; ++k) v[k] = at[k - 2];
    with_coef(KindC<0>{}, min(x0 - 1 + c, nx), [&](const auto& C, f32x2) { grad_weno(C, v, eps2, nz, vl, vr); });
    sl[d * Sh::NX + i] = vl;
    sr[d * Sh::NX + i] = vr;
  }
  __syncthreads();
  for (int it = tid; it < 2 * kGX * kGY; it += kGT) {
    const int d = it / (kGX * kGY), i = it % (kGX * kGY), r = i / kGX, f = i % kGX;
    const int F = x0 + f, y = y0 + r;
    if (F > nx || y >= ny) continue;
    const int o = d * Sh::NX + r * Sh::PX + f;
    fx[((int64_t)d * ny + y) * (nx + 1) + F] = f2_mul(half, f2_add(sr[o], sl[o + 1]));
  }
  __syncthreads();
  // y faces: along the columns
  for (int it = tid; it < 2 * Sh::NY; it += kGT) {
    const int d = it >= Sh::NY, i = d ? it - Sh::NY : it, r = i / kGX, c = i - r * kGX;  // cell y0 - 1 + r
    const f32x2* at = sg + d * Sh::NG + (r + 2) * Sh::GX + c + 3;
    f32x2 v[5], vl, vr;
#pragma unroll
    for (int k = 0; k < 5; ++k) v[k] = at[(k - 2) * Sh::GX];
    with_coef(KindC<1>{}, min(y0 - 1 + r, ny), [&](const auto& C, f32x2) { grad_weno(C, v, eps2, nz, vl, vr); });
    sl[d * Sh::NY + i] = vl;
    sr[d * Sh::NY + i] = vr;
  }
  __syncthreads();
  for (int it = tid; it < 2 * kGX * kGY; it += kGT) {
    const int d = it / (kGX * kGY), i = it % (kGX * kGY), r = i / kGX, c = i % kGX;
    const int F = y0 + r, x = x0 + c;
    if (F > ny || x >= nx) continue;
    const int o = d * Sh::NY + r * kGX + c;
    fy[((int64_t)d * (ny + 1) + F) * nx + x] = f2_mul(half, f2_add(sr[o], sl[o + kGX]));
  }
}

// The velocities of visc_velocities as FP32 (u, v) pairs.
template <int NF>
__global__ void __launch_bounds__(256) visc_velocity_pairs(const DevParams P, const double* __restrict__ q,
                                                          const int ncol, const int nrow, f32x2* __restrict__ vel) {
  const int64_t cells = (int64_t)ncol * nrow;
  const double one = fma64_unit(P.inv_d[0]).one;
  griddep_wait();
  for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < cells; t += (int64_t)gridDim.x * blockDim.x) {
    const int col = (int)(t % ncol), row = (int)(t / ncol);
    bool fx = false, fy = false;
    const int gx = map_cell(col - 5, P.n[0], P.bc_beg[0], P.bc_end[0], &fx);
    const int gy = map_cell(row - 5, P.n[1], P.bc_beg[1], P.bc_end[1], &fy);
    const double* c = q + (int64_t)gy * P.sy + gx;
    double rho = __ldg(c);
#pragma unroll
    for (int f = 1; f < NF; ++f) rho = __fma_rn(rho, one, __ldg(c + f * P.sv));
    // fmax(rho, 1e-16) on the bits, which order like the values of positive
    // numbers (a comparison would occupy the FP64 unit); NaN gives 1e-16 too
    const long long b = __double_as_longlong(rho);
    if (b < __double_as_longlong(1e-16) || b > 0x7ff0000000000000ll) rho = 1e-16;
    const DivisorF64 R = divisor(rho);
    const double mu = __ldg(c + NF * P.sv), mv = __ldg(c + (NF + 1) * P.sv);
    vel[t] = f2_pack(d2f_bits(div_rn(fx ? -mu : mu, R)), d2f_bits(div_rn(fy ? -mv : mv, R)));
  }
}

template <int NF>
cudaError_t launch_tiled(const DevParams& P, const ViscGradBuffers& B, const double* q, cudaStream_t st) {
  const int nx = P.n[0], ny = P.n[1], vcol = nx + 10, vrow = ny + 10;
  const int64_t cells = (int64_t)vcol * vrow;
  cudaError_t e = launch_dependent(&visc_velocity_pairs<NF>, dim3((unsigned)std::min<int64_t>((cells + 255) / 256, 152 * 16)),
                                   dim3(256), 0, st, P, q, vcol, vrow, reinterpret_cast<f32x2*>(B.vel));
  if (e != cudaSuccess) return e;
  const auto kernel = B.uniform.on ? visc_gradients_tiled<true> : visc_gradients_tiled<false>;
  e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)GradShape::kBytes);
  if (e != cudaSuccess) return e;
  // nx + 1 and ny + 1 faces; along x alone, which takes more than 65535 rows of tiles
  const dim3 grid((unsigned)(nx / kGX + 1) * (unsigned)(ny / kGY + 1));
  return launch_dependent(kernel, grid, dim3(kGT), GradShape::kBytes, st, P, B.uniform, B.cf[0], B.cf[1],
                          reinterpret_cast<const f32x2*>(B.vel), reinterpret_cast<f32x2*>(B.fg[0]),
                          reinterpret_cast<f32x2*>(B.fg[1]));
}

template <int ND, int NF, class RT>
cudaError_t launch_all(const DevParams& P, const ViscGradBuffers& B, const double* q, cudaStream_t st) {
  const int nx = P.n[0], ny = ND > 1 ? P.n[1] : 1;
  auto grid = [](int64_t items) { return (unsigned)std::min<int64_t>((items + 255) / 256, 152 * 16); };
  const int vcol = nx + 10, vrow = ND > 1 ? ny + 10 : 1;
  visc_velocities<ND, NF><<<grid((int64_t)vcol * vrow), 256, 0, st>>>(P, q, vcol, vrow, B.vel);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return e;
  // G on x = -3 .. nx+2 (and y = -3 .. ny+2)
  const int gcol = nx + 6, grow = ND > 1 ? ny + 6 : 1, gjb = ND > 1 ? -3 : 0;
  visc_cell_gradients<ND, RT><<<grid((int64_t)gcol * grow), 256, 0, st>>>(P, B, vcol, vrow, -3, gjb, gcol, grow,
                                                                           B.g);
  if ((e = cudaGetLastError()) != cudaSuccess) return e;
  const int64_t xwarps = (int64_t)((nx + 1 + 30) / 31) * ny;
  visc_face_gradients_x<ND, RT><<<grid(32 * xwarps), 256, 0, st>>>(P, B.cf[0], B.g, -3, gjb, gcol, grow, B.fg[0]);
  if ((e = cudaGetLastError()) != cudaSuccess) return e;
  if constexpr (ND > 1) {
    static_assert(sizeof(RT) == 8, "2-D split and gated contexts take launch_tiled");
    constexpr int R = 8;  // faces per thread
    visc_face_gradients_y<R><<<grid((int64_t)nx * ((ny + 1 + R - 1) / R)), 256, 0, st>>>(P, B.g, -3, gjb, gcol, grow,
                                                                                        B.fg[1]);
    e = cudaGetLastError();
  }
  return e;
}

}  // namespace

cudaError_t visc_gradients_launch(int nd, int nf, bool fp32, const DevParams& P, const ViscGradBuffers& B,
                                  const double* q, cudaStream_t st) {
  if (fp32) {
    if (B.cf[0] == nullptr || (nd > 1 && B.cf[1] == nullptr)) return cudaErrorInvalidValue;
    if (nd == 1 && nf == 1) return launch_all<1, 1, float>(P, B, q, st);
    if (nd == 1 && nf == 2) return launch_all<1, 2, float>(P, B, q, st);
    if (nd == 2 && nf == 1) return launch_tiled<1>(P, B, q, st);
    if (nd == 2 && nf == 2) return launch_tiled<2>(P, B, q, st);
  } else {
    if (nd == 1 && nf == 1) return launch_all<1, 1, double>(P, B, q, st);
    if (nd == 1 && nf == 2) return launch_all<1, 2, double>(P, B, q, st);
    if (nd == 2 && nf == 1) return launch_all<2, 1, double>(P, B, q, st);
    if (nd == 2 && nf == 2) return launch_all<2, 2, double>(P, B, q, st);
  }
  return cudaErrorInvalidValue;
}

}  // namespace mfc
