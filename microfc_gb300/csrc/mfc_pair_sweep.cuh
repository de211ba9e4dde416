// The directional sweeps of a split-precision 3-D WENO5 stage: what
// sweep_kernel (mfc_sweep.cuh) does, the same operations in the same order, for
// variables kept in interleaved FP32 pairs everywhere.
//
// A sweep is bound by instruction issue and the latency of its phases (HBM was
// at 3.6, 2.9 and 4.7 TB/s in the x, y and z sweeps).  Hence, as in the 2-D
// pair kernel (mfc_pair.cuh):
//
//   * the primitives and the partial RHS lie in memory as pairs (pair k of
//     cell o at k * sv + o), so a tile arrives by one bulk copy in its final
//     layout, without a conversion loop and its barrier, and every access of
//     every phase is 64 bits wide, in the y and z sweeps with x across the
//     lanes and no bank conflicts;
//   * the z sweep converts the state it makes, in registers, and stores the
//     pairs for the next stage (PrimPairs), whose x sweep then loads 32 bytes
//     a cell and converts nothing; without them (a new state) the x sweep
//     converts and stores them for the other two;
//   * a thread reconstructs a run of R = 9 cells of one pencil and pair: 13
//     loads instead of 45, one difference a cell instead of four.  16 pencils
//     x 2 runs x 4 pairs are the block's 128 threads;
//   * a face's fluxes and interface velocity overwrite the right values they
//     come from: 30-31 KB a block of 128 threads, seven blocks on an SM.
//
// Measured at 256^3 (us a stage: x, y, z sweep; before: sweep_kernel): 591,
// 558, 672 to 815 -> 389, 392, 668 to 872 (the z sweep at 5.7 to 6.0 TB/s, with
// the pairs it stores; the others at 68 % issue); a step 5717 -> 4799.  With
// the x sweep's pairs by plain loads 5012; registers uncapped, 5 % slower.
#pragma once

#include "mfc_device.cuh"
#include "mfc_stage.cuh"
#include "mfc_sweep.cuh"
#include "mfc_tma.cuh"

namespace mfc {

// DIR 0 keeps [pair][row][cell of the sweep]; its tile rows start one cell
// before the halo and end one after, on the 16 bytes a bulk copy asks for.
template <int NF, int DIR, int TA, int TB>
struct PairSweepShape {
  using Q = Eqs<3, NF>;
  static constexpr int S = Q::S, H = 3, NPR = S / 2, LA = TA + 2 * H, NCA = TA + 2;
  static constexpr int LEAD = DIR == 0 ? 1 : 0, PLA = DIR == 0 ? LA + 2 : LA;
  static_assert(S % 2 == 0, "3-D pairs need an even number of variables");
  static constexpr int NQ = NPR * PLA * TB, NW = NPR * NCA * TB;
  static constexpr size_t kBarOffset = sizeof(f32x2) * size_t(NQ + 2 * NW);
  static constexpr size_t kCoefOffset = kBarOffset + 16;
  static constexpr size_t kCoefBytes = sizeof(float) * size_t(kCoefRec) * NCA;  // not used on a uniform grid
  static constexpr uint32_t kBoxBytes = uint32_t(sizeof(f32x2)) * NQ;
};

// T maps B.cur (T.on = 0: plain loads only).
template <int NF, int DIR, int TA, int TB, int NT, int R, bool TMA, int MINB>
__global__ void __launch_bounds__(NT, MINB) pair_sweep_kernel(const DevParams P, const __grid_constant__ UniformCoef U,
                                                              const __grid_constant__ TileMap T,
                                                              const double* __restrict__ qin,
                                                              const double* __restrict__ qbase,
                                                              double* __restrict__ qout, const double dt,
                                                              const int kind, const PrimPairs B) {
  using Sh = PairSweepShape<NF, DIR, TA, TB>;
  using Q = Eqs<3, NF>;
  constexpr int S = Sh::S, H = Sh::H, NPR = Sh::NPR, LA = Sh::LA, NCA = Sh::NCA, PLA = Sh::PLA;
  constexpr int SA = DIR == 0 ? 1 : TB;  // the sweep's step in shared memory
  extern __shared__ __align__(128) unsigned char smem_pair[];
  f32x2* const sq = reinterpret_cast<f32x2*>(smem_pair);  // [pair][LA][TB], DIR 0: [pair][TB][PLA]
  f32x2* const wl = sq + Sh::NQ;                           // [pair][NCA][TB], DIR 0: [pair][TB][NCA]
  f32x2* const wr = wl + Sh::NW;
  float* const sc = reinterpret_cast<float*>(smem_pair + Sh::kCoefOffset);
  auto qi = [](int pr, int la, int p) { return DIR == 0 ? (pr * TB + p) * PLA + la + Sh::LEAD : (pr * LA + la) * TB + p; };
  auto wi = [](int pr, int ca, int p) { return DIR == 0 ? (pr * TB + p) * NCA + ca : (pr * NCA + ca) * TB + p; };
  // pair k of the results of face f (left of tile cell f): the fluxes, then the
  // interface velocity, in the right-value slots and left-value slot 0
  auto fl = [&](int k, int f, int p) -> f32x2& { return k < NPR ? wr[wi(k, f, p)] : wl[wi(k - NPR, f + 1, p)]; };
  auto prim = [&](int v, int la, int p) { return reinterpret_cast<const float*>(sq)[qi(v >> 1, la, p) * 2 + (v & 1)]; };

  const int tid = threadIdx.x;
  // pencils lie along y (x sweep) or x
  const int b0 = (DIR == 0 ? blockIdx.y : blockIdx.x) * TB, a0 = (DIR == 0 ? blockIdx.x : blockIdx.y) * TA;
  const int gc = blockIdx.z, na = P.n[DIR], nb = P.n[DIR == 0 ? 1 : 0];
  const int64_t sa = DIR == 0 ? 1 : DIR == 1 ? P.sy : P.sz, sb = DIR == 0 ? P.sy : 1;
  const int64_t oc = gc * (DIR == 2 ? P.sy : P.sz);  // cell (a, b) of the block: oc + a * sa + b * sb
  const double one = fma64_unit(P.inv_d[0]).one;     // the FP64 sums' register operand
  float gam_i[NF], pi_i[NF];
#pragma unroll
  for (int f = 0; f < NF; ++f) {
    gam_i[f] = P.gammas_f[f];
    pi_i[f] = P.pi_infs_f[f];
  }
  const bool uni = U.on[DIR] != 0;
  f32x2* const grhs = reinterpret_cast<f32x2*>(P.work);  // partial RHS pairs

  for (int it = uni ? kCoefRec * NCA : tid; it < kCoefRec * NCA; it += NT) {
    const int ca = it % NCA, k = it / NCA;
    sc[ca * kCoefRec + k] =
        k < kNumCoef ? d2f_bits(__ldg(P.coef[DIR] + k * P.cstride[DIR] + clamp_coef_index(a0 - 1 + ca, na) + P.coff))
                     : 0.f;
  }
  bool use_tma = false;
  uint32_t bar = 0;
  if constexpr (TMA) {
    use_tma = T.on && (DIR > 0 || B.in != nullptr) && a0 >= H && a0 + TA + H <= na && b0 + TB <= nb;
    if (use_tma) {
      bar = smem_addr(smem_pair + Sh::kBarOffset);
      if (tid == 0) mbar_init(bar, 1);
    }
  }
  griddep_wait();  // the state, the primitives and the partial RHS are earlier kernels' output
  // The operands of the last phase that the tile load does not bring in: the
  // partial RHS and, on the z sweep, the RK registers, every 128-byte line
  // (16 cells of a row) prefetched into L2 while the tile is worked on: at
  // 256^3 a register is 1 GB and none of them stays in L2 between the sweeps.
  if constexpr (DIR > 0) {
    static_assert(TB == 16, "a row of the tile is one 128-byte line");
    const int nreg = DIR == 1 || kind == kRhsOnly ? 0 : (kind == kRkEuler ? 1 : 2);
    for (int it = tid; it < TA * (NPR + nreg * S); it += NT) {
      const int ta = it % TA, r = it / TA, ga = a0 + ta;
      if (ga >= na) continue;
      const int64_t o = oc + ga * sa + b0;
      const void* ptr = r < NPR ? static_cast<const void*>(grhs + o + r * P.sv)
                        : r < NPR + S ? static_cast<const void*>(qbase + o + (r - NPR) * P.sv)
                                      : static_cast<const void*>(qin + o + (r - NPR - S) * P.sv);
      asm volatile("prefetch.global.L2 [%0];" ::"l"(ptr));
    }
  }
  if (use_tma) {
    volatile int* landed = reinterpret_cast<volatile int*>(smem_pair + Sh::kBarOffset + 8);
    if (tid == 0) {
      mbar_arrive_expect_tx(bar, Sh::kBoxBytes);
      if (DIR == 0) tma_load_4d(smem_addr(sq), &T.map, a0 - H - Sh::LEAD, b0, gc, 0, bar);
      else if (DIR == 1) tma_load_4d(smem_addr(sq), &T.map, b0, a0 - H, gc, 0, bar);
      else tma_load_4d(smem_addr(sq), &T.map, b0, gc, a0 - H, 0, bar);
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
  } else {  // plain loads, with the boundary conditions and processor halos
    // thread order: x fastest, for coalesced loads
    for (int it = tid; it < TB * LA; it += NT) {
      const int p = DIR == 0 ? it / LA : it % TB, la = DIR == 0 ? it % LA : it / TB, ra = a0 - H + la;
      bool fa = false, fb = false;
      const int gb = map_cell(b0 + p, nb, P.bc_beg[DIR == 0 ? 1 : 0], P.bc_end[DIR == 0 ? 1 : 0], &fb);
      const int ga = map_cell(ra, na, P.bc_beg[DIR], P.bc_end[DIR], &fa);
      const int64_t o = oc + ga * sa + gb * sb;
      // processor boundary along the sweep: the ghost cell comes, as
      // conservative values, from the neighbour's halo buffer (x: [S][nz][ny][H],
      // y: [S][nz][H][nx], z: [S][H][ny][nx]; depth 0 next to the boundary)
      const int side = ra < 0 ? (P.bc_beg[DIR] >= 0 ? 0 : -1) : (ra >= na && P.bc_end[DIR] >= 0 ? 1 : -1);
      if (side < 0 && (DIR > 0 || B.in != nullptr)) {
        f32x2 w[NPR];
#pragma unroll
        for (int k = 0; k < NPR; ++k) w[k] = __ldg(B.cur + o + k * P.sv);
        // a reflected cell's normal velocity negated: the conversion is odd in the momentum
        if (fa) w[(Q::MOM + DIR) / 2] ^= 0x80000000ull << ((Q::MOM + DIR) % 2 * 32);
#pragma unroll
        for (int k = 0; k < NPR; ++k) sq[qi(k, la, p)] = w[k];
        continue;
      }
      const double* src = qin + o;
      int64_t vs = P.sv;
      if (side >= 0) {
        const int d = min(side == 0 ? -1 - ra : ra - na, H - 1);  // deeper cells of partial tiles are never stored
        const int64_t nx = P.n[0], ny = P.n[1], nz = P.n[2];
        const int64_t at = DIR == 0 ? (gc * ny + gb) * H + d : DIR == 1 ? ((int64_t)gc * H + d) * nx + gb : (d * ny + gc) * nx + gb;
        src = P.halo[2 * DIR + side] + at;
        vs = H * (DIR == 0 ? nz * ny : DIR == 1 ? nz * nx : ny * nx);
      }
      double q[S];
#pragma unroll
      for (int v = 0; v < S; ++v) q[v] = __ldg(src + v * vs);
      if (side < 0 && fa) q[Q::MOM + DIR] = -q[Q::MOM + DIR];
      float pr[S];
      cons_to_prim_split<3, NF>(q, P, one, pr);
      // a state that came without pairs: this block's cells, for the other sweeps
      const bool own = DIR == 0 && la >= H && la < H + TA && ra < na && b0 + p < nb;
#pragma unroll
      for (int k = 0; k < NPR; ++k) {
        const f32x2 w = f2_pack(pr[2 * k], pr[2 * k + 1]);
        sq[qi(k, la, p)] = w;
        if (own) B.cur[o + k * P.sv] = w;
      }
    }
    __syncthreads();
  }

  // ---- WENO along the sweep for cells a0-1 .. a0+TA --------------------------------
  {
    static_assert(NCA % R == 0, "runs must fill the pencils");
    const f32x2 eps2 = f2_pack(P.weno_eps_f, P.weno_eps_f);
    auto runs = [&](auto uni_c) {
      for (int it = tid; it < NPR * TB * (NCA / R); it += NT) {
        // x sweep: the runs of a row side by side, so that 16 lanes, on eight
        // rows, meet in pairs of banks at most four times on loads and never
        // on stores (rows of 24 and 18 pairs)
        constexpr int RUNS = NCA / R;
        const int p = DIR == 0 ? it / RUNS % TB : it % TB, q = it / TB;
        const int w = DIR == 0 ? it / (RUNS * TB) : q % NPR, c0 = (DIR == 0 ? it % RUNS : q / NPR) * R;
        const f32x2* at = sq + qi(w, c0 + H - 1, p);
        f32x2* l = wl + wi(w, c0, p);
        f32x2* r = wr + wi(w, c0, p);
        f32x2 v1 = at[-SA], v2 = at[0], v3 = at[SA];
        f32x2 dm2 = f2_sub(v1, at[-2 * SA]), dm1 = f2_sub(v2, v1), d0 = f2_sub(v3, v2);
#pragma unroll 3
        for (int j = 0; j < R; ++j) {
          const f32x2 v4 = at[(j + 2) * SA], d1 = f2_sub(v4, v3);
          f32x2 vl, vr;
          if constexpr (decltype(uni_c)::value) {
            weno5_pair_diffs([&](int k) { return f32x2(U.rec[DIR][k]); }, v2, d1, d0, dm1, dm2, eps2, vl, vr);
          } else {
            float c[kCoefRec];
            load_coef_record(sc + (c0 + j) * kCoefRec, c);
            weno5_pair_diffs([&](int k) { return f2_pack(c[k], c[k]); }, v2, d1, d0, dm1, dm2, eps2, vl, vr);
          }
          l[j * SA] = vl;
          r[j * SA] = vr;
          v2 = v3;
          v3 = v4;
          dm2 = dm1;
          dm1 = d0;
          d0 = d1;
        }
      }
    };
    if (uni) runs(FlagC<true>{});
    else runs(FlagC<false>{});
  }
  __syncthreads();

  // ---- HLLC on faces a0-1/2 .. a0+TA-1/2 ---------------------------------------------
  for (int it = tid; it < TB * (TA + 1); it += NT) {
    const int p = DIR == 0 ? it / (TA + 1) : it % TB, f = DIR == 0 ? it % (TA + 1) : it / TB, gface = a0 - 1 + f;
    const bool lfr = gface == -1 && P.bc_beg[DIR] == -4, rfl = gface == na - 1 && P.bc_end[DIR] == -4;
    float qL[S], qR[S], F[S], us;
#pragma unroll
    for (int k = 0; k < NPR; ++k) {
      const f32x2 a = wr[wi(k, f, p)], b = wl[wi(k, f + 1, p)];
      f2_unpack(lfr ? b : a, qL[2 * k], qL[2 * k + 1]);
      f2_unpack(rfl ? a : b, qR[2 * k], qR[2 * k + 1]);
    }
    hllc_face_fast<3, NF, DIR>(qL, qR, gam_i, pi_i, F, us);
#pragma unroll
    for (int k = 0; k < NPR; ++k) fl(k, f, p) = f2_pack(F[2 * k], F[2 * k + 1]);
    fl(NPR, f, p) = f2_pack(us, 0.f);
  }
  __syncthreads();

  // ---- flux divergence, accumulation, RK on the last sweep ---------------------------
  griddep_launch_dependents();
  bool bad = false, nonphys = false;
  double icfl = 0.0;
  const float dtf = __double2float_rn(dt);  // the increments are FP32
  // KIND: the stage's combination as a compile-time constant, chosen once per block
  auto finish = [&](auto kind_c) {
    constexpr int KIND = decltype(kind_c)::value;
    for (int it = tid; it < TB * TA; it += NT) {
      const int p = DIR == 0 ? it / TA : it % TB, ta = DIR == 0 ? it % TA : it / TB, ga = a0 + ta, gb = b0 + p;
      if (ga >= na || gb >= nb) continue;
      const int64_t o = oc + ga * sa + gb * sb;
      f32x2 part[NPR];
      double base[S], in[S];  // all loads in flight before the divergence
#pragma unroll
      for (int k = 0; k < NPR; ++k) part[k] = DIR == 0 ? 0 : grhs[o + k * P.sv];
      if constexpr (DIR == 2 && KIND != kRhsOnly) {
#pragma unroll
        for (int v = 0; v < S; ++v) base[v] = __ldg(qbase + o + v * P.sv);
        if constexpr (KIND != kRkEuler) {
#pragma unroll
          for (int v = 0; v < S; ++v) in[v] = __ldg(qin + o + v * P.sv);
        }
      }
      const float inv = d2f_bits(__ldg(P.inv_d[DIR] + ga));
      float r[S];
#pragma unroll
      for (int k = 0; k < NPR; ++k) {
        float d0, d1, r0, r1;
        f2_unpack(f2_sub(fl(k, ta, p), fl(k, ta + 1, p)), d0, d1);
        f2_unpack(part[k], r0, r1);
        r[2 * k] = DIR == 0 ? inv * d0 : mul_add(inv, d0, r0);
        r[2 * k + 1] = DIR == 0 ? inv * d1 : mul_add(inv, d1, r1);
      }
      float u0, u1, pad;
      f2_unpack(fl(NPR, ta, p), u0, pad);
      f2_unpack(fl(NPR, ta + 1, p), u1, pad);
      const float du = u1 - u0;
#pragma unroll
      for (int f = 0; f < NF; ++f) {
        const float a = prim(Q::ADV + f, ta + H, p);
        r[Q::ADV + f] = mul_add(inv * a, du, r[Q::ADV + f]);
      }
      if constexpr (DIR < 2) {
#pragma unroll
        for (int k = 0; k < NPR; ++k) grhs[o + k * P.sv] = f2_pack(r[2 * k], r[2 * k + 1]);
      } else {
        double out[S];
#pragma unroll
        for (int v = 0; v < S; ++v) {
          if constexpr (KIND == kRhsOnly) out[v] = f2d_bits(r[v]);
          else out[v] = rk_combine_split(KIND, base[v], KIND == kRkEuler ? base[v] : in[v], dtf, r[v], one);
          bad |= not_finite(out[v]);
          qout[o + v * P.sv] = out[v];
        }
        if (KIND != kRhsOnly && B.out != nullptr) {  // the next stage's primitives
          float pr[S];
          cons_to_prim_split<3, NF>(out, P, one, pr);
#pragma unroll
          for (int k = 0; k < NPR; ++k) B.out[o + k * P.sv] = f2_pack(pr[2 * k], pr[2 * k + 1]);
        }
      }
    }
  };
  if constexpr (DIR < 2) {
    finish(KindC<kRhsOnly>{});  // stores the partial RHS whatever the kind
  } else {
    switch (kind) {
      case kRkEuler: finish(KindC<kRkEuler>{}); break;
      case kRk2Final: finish(KindC<kRk2Final>{}); break;
      case kRk3Mid: finish(KindC<kRk3Mid>{}); break;
      case kRk3Final: finish(KindC<kRk3Final>{}); break;
      default: finish(KindC<kRhsOnly>{}); break;
    }
    // the stability monitor (the last stage of a monitored step) reads the
    // new state back: this thread's own stores, from L1
    if (P.monitor) {
      for (int it = tid; it < TB * TA; it += NT) {
        const int p = it % TB, ta = it / TB, ga = a0 + ta, gx = b0 + p;
        if (ga >= na || gx >= nb) continue;
        const int64_t o = oc + ga * sa + gx;
        double qn[S];
#pragma unroll
        for (int v = 0; v < S; ++v) qn[v] = qout[o + v * P.sv];
        const double inv[3] = {__ldg(P.inv_d[0] + gx), __ldg(P.inv_d[1] + gc), __ldg(P.inv_d[2] + ga)};
        bool np;
        const double c = cell_icfl<3, NF>(qn, P, dt, inv, np);
        nonphys |= np;
        if (!(c <= icfl)) icfl = c;  // keeps NaN
      }
      monitor_max(P.monitor, icfl);
    }
    if (bad && P.status) atomicOr(P.status, MFC_FLAG_NAN);
    if (nonphys && P.status) atomicOr(P.status, MFC_FLAG_NEG_PRESSURE);
  }
}

}  // namespace mfc
