// mcv_strip64.cuh -- the stage kernel in strip form, FP64 throughout: the
// layout and the march of mcv_strip.cuh (a warp owns up to 29 cells of a cell
// row and marches along y, lane l holding the H x H points of cell column
// c0 - 1 + l), with the metric read from the caller's planes.
//
// Every quantity is a double, so a lane's cell takes most of its registers and
// its staged rows most of shared memory: MCV4 runs four warps per SM, each with
// a strip twice as long as split precision's.  Derivatives are per cell (times
// dx); the stage weights carry the 1/dx.  phi is advanced as phi + rsg (...)
// with rsg = 1/sqrtG from a plane computed with the geometry, and the Coriolis
// term takes sqrtG f from another: sqrtG (vort + f) = (dvdx - dudy) + sqrtG f.
//
// Compiled without FMA contraction: every instantiation gives the same bits.
#pragma once
#include "mcv_strip.cuh"

namespace mcv {

// Shared memory of one warp for stage kind KIND.
template <int D, int KIND>
struct Strip64Smem {
  static constexpr int H = D - 1;
  static constexpr int RP = 32 * H;  // points of a warp's row
  static constexpr int RE = RP + 4;  // staged elements (a box starts at a multiple of 4)
  static constexpr bool RK3 = KIND == RK3_S2 || KIND == RK3_S3;                       // the update reads the stage input
  static constexpr bool ACC_IN = KIND == RK4_S2 || KIND == RK4_S3 || KIND == RK4_S4;  // ... the RK4 sum
  static constexpr bool ACC_OUT = KIND == RK4_S1 || KIND == RK4_S2 || KIND == RK4_S3;
  static constexpr int FB = (int)align128((size_t)H * RE * 8);  // one staged field of a cell row
  static constexpr int PT = H * H * 32 * 8;                     // one double per point of the lanes' cells
  static constexpr int IN = 0;               // u, v, phi, phi_s, sqrtG, G^11, G^12, G^22
  static constexpr int RS = IN + 8 * FB;     // 1/sqrtG, sqrtG f of the cell row to update
  static constexpr int OUT = RS + 2 * FB;    // its RK base; the results take its place
  static constexpr int ACC = OUT + 3 * FB;   // RK4 sums
  static constexpr int AR = ACC + ((ACC_IN || ACC_OUT) ? 3 * FB : 0);  // x sweep: fx, dx, dvdx, cU (RK3: and v)
  static constexpr int NA = RK3 ? 5 : 4;
  static constexpr int CV = AR + NA * PT;    // cV, two slots
  static constexpr int BAR = CV + 2 * PT;
  static constexpr int BYTES = (int)align128(BAR + 16);
  static_assert(NA * PT + 2 * PT >= 8 * RE * 8, "the strip's first row is staged over the sweep results");
  // warps per block, one block per SM: shared memory (227 KB) and registers
  static constexpr int WMAX = D == 3 ? 8 : 4;
  static constexpr int WPB = 232448 / BYTES < WMAX ? 232448 / BYTES : WMAX;
};

// One-sided derivatives of a line from its points (src/spatial_operators_mod.F90:204-238), per cell.
template <int D>
__device__ __forceinline__ double end_left(const double *p) {
  if constexpr (D == 3) return __fma_rn(-3., p[0], __fma_rn(4., p[1], -p[2]));
  else return __fma_rn(-5.5, p[0], __fma_rn(9., p[1], __fma_rn(-4.5, p[2], p[3])));
}
template <int D>
__device__ __forceinline__ double end_right(const double *p) {
  if constexpr (D == 3) return __fma_rn(3., p[2], __fma_rn(-4., p[1], p[0]));
  else return __fma_rn(5.5, p[3], __fma_rn(-9., p[2], __fma_rn(4.5, p[1], -p[0])));
}
// The interior points of a cell (:179-200): the part without the right end's, and that.
template <int D>
__device__ __forceinline__ void interior64(double o0, const double *c, double &b1, double &b2) {
  const double via = c[D - 1] - c[0];
  if constexpr (D == 3) {
    b1 = __fma_rn(1.5, via, -0.25 * o0);
    b2 = 0.;
  } else {
    const double k = (2. / 3.) * ((c[0] + c[3]) - (c[1] + c[2]));
    b1 = __fma_rn(-4. / 27., o0, __fma_rn(4. / 3., via, -k));
    b2 = __fma_rn(-5. / 27., o0, __fma_rn(4. / 3., via, k));
  }
}
template <int D>
__device__ __forceinline__ double interior64_end1(double b1, double o3) {
  return __fma_rn(D == 3 ? -0.25 : -5. / 27., o3, b1);
}
__device__ __forceinline__ double interior64_end2(double b2, double o3) { return __fma_rn(-4. / 27., o3, b2); }

template <int D, int KIND, int NB, bool IDENT>
__global__ void __launch_bounds__(32 * Strip64Smem<D, KIND>::WPB, 1)
    strip64_kernel(const __grid_constant__ StageBatch<NB> b) {
  using S = Strip64Smem<D, KIND>;
  constexpr int H = D - 1, RE = S::RE, WPB = S::WPB, FE = S::FB / 8, PE = S::PT / 8;
  constexpr unsigned ALL = 0xffffffffu;
  // weights of the RK base and the stage input in the update (src/time_scheme_mod.F90:60-123)
  constexpr double KB = KIND == RK3_S2 ? 0.75 : KIND == RK3_S3 ? 1. / 3. : 1.;
  constexpr double KU = KIND == RK3_S2 ? 0.25 : 2. / 3.;
  extern __shared__ __align__(128) unsigned char smraw[];
  const int lane = threadIdx.x & 31;
  const int warp = __shfl_sync(ALL, (int)(threadIdx.x >> 5), 0);  // uniform, and known to be
  unsigned char *sm = smraw + warp * S::BYTES;
  double *in = reinterpret_cast<double *>(sm + S::IN);
  double *ar = reinterpret_cast<double *>(sm + S::AR) + lane;
  double *cvs = reinterpret_cast<double *>(sm + S::CV) + lane;
  uint64_t *bar = reinterpret_cast<uint64_t *>(sm + S::BAR);  // [0] the input, [1] the update's operands
  if (lane == 0) {
    mbar_init(bar, 1);
    mbar_init(bar + 1, 1);
    fence_mbar_init();
  }
  __syncwarp();
  uint32_t par0 = 0, par1 = 0;
  bool waited = false;
  const int stride = gridDim.x * WPB;

  // runs are dealt to the blocks in turn, so that few of them use every SM
  for (int id = warp * gridDim.x + blockIdx.x; id < b.total; id += stride) {
  int x, xe;
  strip_work(b, id, x, xe);
  while (x < xe) {
    int k;
    Strip st;
    if (!next_strip(b, id, x, xe, k, st)) continue;
    const GridDesc &g = b.g[k];
    const StageArgs &a = b.a[k];
    const TileMaps &tm = b.tm[k];
    const int c0 = st.c0, w = st.w, r0 = st.r0, r1 = st.r1, panel = st.panel;
    const int mem = IDENT ? st.slot : active_member(a.active, a.ident, st.slot);
    const int X0 = c0 * H;  // padded index of lane 0's first point
    const int X0a = X0 & ~3, rem = X0 - X0a;
    const long long pbase = (long long)panel * g.plane, fbase = (long long)mem * g.mstride + pbase;
    const int P = g.P;
    const double inc = a.inc * g.inv_dx, sfx = g.dx;  // tendencies come times dx
    if (id + stride >= b.total && x >= xe) allow_dependent_launch();
    if (!waited) {
      wait_prerequisite_grid();  // the halo kernel before
      waited = true;
    }

    // ---- copies (one lane).  Cell row c's rows: padded (c + 1) H + 1 .. (c + 2) H.
    const int frow = (mem * 6 + panel) * g.np, prow = panel * g.np;
    constexpr uint32_t BB = H * RE * 8;
    auto issue_in = [&](int c) {
      const int row = (c + 1) * H + 1;
#pragma unroll
      for (int f = 0; f < 8; ++f)
        tma_load_2d(sm + S::IN + f * S::FB, &tm.f[f], X0a, (f < 4 ? frow : prow) + row, bar);
    };
    constexpr uint32_t UP_BYTES = (5 + (S::ACC_IN ? 3 : 0)) * BB;
    auto issue_up = [&](int c) {
      const int row = (c + 1) * H + 1;
      mbar_arrive_expect_tx(bar + 1, UP_BYTES);
#pragma unroll
      for (int f = 0; f < 2; ++f) tma_load_2d(sm + S::RS + f * S::FB, &tm.f[8 + f], X0a, prow + row, bar + 1);
#pragma unroll
      for (int f = 0; f < 3; ++f) tma_load_2d(sm + S::OUT + f * S::FB, &tm.f[10 + f], X0a, frow + row, bar + 1);
      if constexpr (S::ACC_IN) {
#pragma unroll
        for (int f = 0; f < 3; ++f) tma_load_2d(sm + S::ACC + f * S::FB, &tm.f[13 + f], X0a, frow + row, bar + 1);
      }
    };
    // Bounded wait for the copies of barrier i; false: give up (the copies in flight have landed or the
    // limit has run out twice).
    auto wait_for = [&](int i, uint32_t parity) {
      bool ok = mbar_try_wait(bar + i, parity);
      if (!__all_sync(ALL, ok)) {
        if (!ok) ok = mbar_wait_bounded(bar + i, parity);
        if (!__all_sync(ALL, ok)) {
          if (lane == 0) *(volatile int *)a.err = 1;
          mbar_wait_bounded(bar, par0);
          mbar_wait_bounded(bar + 1, par1);
          return false;
        }
      }
      return true;
    };

    // pointwise quantities of one staged row (fields fs apart; spatial_operators_mod.F90:58-61), the
    // interface wave speeds |c| + sqrt(G^ii phi) (:248-280) in x at the cell's first point and, for a row
    // of interface points, in y (the sign bit says cV < 0, which a wind of -0 is not and a speed that is
    // not a number does not hide)
    struct Row {
      double e[H], u[H], v[H], pg[H], cu[H], lx;
    };
    auto row_values = [&](const double *f, int fs, Row &o, double *cv, int cvst, double *ly) {
      const int at = rem + lane * H;
      double p[8][H];
#pragma unroll
      for (int x = 0; x < 8; ++x) lane_load<H>(f + x * fs + at, p[x]);
#pragma unroll
      for (int i = 0; i < H; ++i) {
        const double u = p[0][i], v = p[1][i], ph = p[2][i], g11 = p[5][i], g12 = p[6][i], g22 = p[7][i];
        const double cu = __fma_rn(g12, v, g11 * u);  // cov2contrav, projection_mod.F90:138-148
        const double cw = __fma_rn(g22, v, g12 * u);
        o.u[i] = u;
        o.v[i] = v;
        o.e[i] = __fma_rn(0.5, __fma_rn(cw, v, cu * u), ph + p[3][i]);  // E = phi + phi_s + K
        o.pg[i] = ph * p[4][i];
        o.cu[i] = cu;
        cv[i * cvst] = cw;
        if (i == 0) o.lx = fabs(cu) + sqrt(g11 * ph);
        if (ly) ly[i] = copysign(fabs(cw) + sqrt(g22 * ph), cw < 0. ? -1. : 1.);
      }
    };

    // ---- carried along y, per column of the lane: the last row's values and the previous cell's
    // top-end derivatives (f + lam q of the flux pairs) and interior parts
    double e0[H], u0[H], v0[H], q0[H], m0[H], lam0[H], sE[H], sM[H], rU[H];
    double bE1[H], bE2[H], bM1[H], bM2[H], bU1[H], bU2[H];

    hand_to_copies();
    if (elect_one()) {
      // the first row of the lower halo cell, then its block
      const int row = r0 * H, nel = min(RE, P - X0a);
      const long long o = (long long)row * P + X0a;
      double *fr = reinterpret_cast<double *>(sm + S::AR);
      const double *src[8] = {a.us + fbase, a.vs + fbase, a.ps + fbase, a.phis + fbase,
                              a.sqrtG + pbase, a.ig11 + pbase, a.ig12 + pbase, a.ig22 + pbase};
      mbar_arrive_expect_tx(bar, 8 * BB + (uint32_t)nel * 64);
#pragma unroll
      for (int f = 0; f < 8; ++f) bulk_load(fr + f * RE, src[f] + o, nel * 8, bar);
      issue_in(r0 - 1);
      issue_up(r0 - 1);
    }
    __syncwarp();
    if (!wait_for(0, par0)) return;
    par0 ^= 1u;
    {
      Row o;
      double cv[H];
      row_values(reinterpret_cast<double *>(sm + S::AR), RE, o, cv, 1, nullptr);
#pragma unroll
      for (int i = 0; i < H; ++i) {
        e0[i] = o.e[i];
        u0[i] = o.u[i];
        v0[i] = o.v[i];
        q0[i] = o.pg[i];
        m0[i] = o.pg[i] * cv[i];
        lam0[i] = sE[i] = sM[i] = rU[i] = 0.;
        bE1[i] = bE2[i] = bM1[i] = bM2[i] = bU1[i] = bU2[i] = 0.;
      }
      __syncwarp();
    }
    const bool last_x = c0 + w == g.Nc;
    const int cnt = w * H + (last_x ? 1 : 0);  // owned points of a row

    for (int c = r0 - 1; c <= r1; ++c) {
      // ---- rows c H + 1 .. c H + H (interior indices) of the lane's cell
      Row o[H];
      double ly[H];
      double *cvc = cvs + (c & 1) * PE, *cvp = cvs + ((c & 1) ^ 1) * PE;  // cV of this cell row, and of the one before
#pragma unroll
      for (int rr = 0; rr < H; ++rr)
        row_values(in + rr * RE, FE, o[rr], cvc + rr * H * 32, 32, rr == H - 1 ? ly : nullptr);
      hand_to_copies();
      if (c < r1) {
        if (elect_one()) {
          mbar_arrive_expect_tx(bar, 8 * BB);
          issue_in(c + 1);
        }
        __syncwarp();
      }
      if (c >= r0)
        if (!wait_for(1, par1)) return;

      // ---- y sweep (:95-125) of the lane's columns: the fluxes at the bottom of cell c, which complete
      // rows (c - 1) H + 1 .. c H of cell c - 1; their tendencies (:127-131) and RK stage update
      constexpr int NP = H == 2 ? 2 : 1;  // points updated at once
      double t[H][3][NP], rsg[H][NP], sf[H][NP];
#pragma unroll
      for (int i = 0; i < H; ++i) {
        double f[D], gE, gM, gU, lE, rE, lV, rV, b1, b2;
        // E with Riemann on v
        f[0] = v0[i];
#pragma unroll
        for (int m = 1; m < D; ++m) f[m] = o[m - 1].v[i];
        lV = end_left<D>(f);
        rV = end_right<D>(f);
        v0[i] = f[H];
        f[0] = e0[i];
#pragma unroll
        for (int m = 1; m < D; ++m) f[m] = o[m - 1].e[i];
        lE = end_left<D>(f);
        rE = end_right<D>(f);
        e0[i] = f[H];
        const double lam = fabs(lam0[i]), lamt = fabs(ly[i]);
        gE = 0.5 * (sE[i] + __fma_rn(-lam, lV, lE));
        sE[i] = __fma_rn(lamt, rV, rE);
        double yE[H], yM[H], yU[H];
        yE[0] = interior64_end1<D>(bE1[i], gE);
        if constexpr (D == 4) yE[1] = interior64_end2(bE2[i], gE);
        yE[H - 1] = gE;
        interior64<D>(gE, f, bE1[i], bE2[i]);
        // phiG cV with Riemann on phiG
        f[0] = q0[i];
#pragma unroll
        for (int m = 1; m < D; ++m) f[m] = o[m - 1].pg[i];
        lV = end_left<D>(f);
        rV = end_right<D>(f);
        q0[i] = f[H];
        f[0] = m0[i];
#pragma unroll
        for (int m = 1; m < D; ++m) f[m] = o[m - 1].pg[i] * cvc[((m - 1) * H + i) * 32];
        lE = end_left<D>(f);
        rE = end_right<D>(f);
        m0[i] = f[H];
        gM = 0.5 * (sM[i] + __fma_rn(-lam, lV, lE));
        sM[i] = __fma_rn(lamt, rV, rE);
        yM[0] = interior64_end1<D>(bM1[i], gM);
        if constexpr (D == 4) yM[1] = interior64_end2(bM2[i], gM);
        yM[H - 1] = gM;
        interior64<D>(gM, f, bM1[i], bM2[i]);
        // dudy, upwinded by cV (:83-85)
        f[0] = u0[i];
#pragma unroll
        for (int m = 1; m < D; ++m) f[m] = o[m - 1].u[i];
        lE = end_left<D>(f);
        gU = __double2hiint(lam0[i]) < 0 ? lE : rU[i];
        rU[i] = end_right<D>(f);
        u0[i] = f[H];
        yU[0] = interior64_end1<D>(bU1[i], gU);
        if constexpr (D == 4) yU[1] = interior64_end2(bU2[i], gU);
        yU[H - 1] = gU;
        interior64<D>(gU, f, b1, b2);
        bU1[i] = b1;
        bU2[i] = b2;
        lam0[i] = ly[i];
        if (c >= r0) {
#pragma unroll
          for (int rr = 0; rr < H; ++rr) {
            const int pt = (rr * H + i) * 32;
            const double cu = ar[3 * PE + pt], cv = cvp[pt];
            // MCV4 is updated point by point, MCV3 both points of the lane at once
            constexpr int N = NP;
            const int at = rr * RE + rem + lane * H + (N == 2 ? 0 : i);
            const double *rs = reinterpret_cast<const double *>(sm + S::RS) + at;
            if (N == 1 || i == 0) {
              lane_load<N>(rs, rsg[rr]);
              lane_load<N>(rs + FE, sf[rr]);
            }
            const int q = N == 2 ? i : 0;
            const double ab = __fma_rn(sfx, sf[rr][q], ar[2 * PE + pt] - yU[rr]);
            const double fx = ar[pt], dx = ar[PE + pt];
            // RK3: the update without its base; fx and dx already hold KU u - inc fx and KU phiG - inc dx
            if constexpr (S::RK3) {
              t[rr][0][q] = __fma_rn(inc, ab * cv, fx);
              t[rr][1][q] = __fma_rn(-inc, __fma_rn(ab, cu, yE[rr]), KU * ar[4 * PE + pt]);
              t[rr][2][q] = rsg[rr][q] * __fma_rn(-inc, yM[rr], dx);
            } else {
              t[rr][0][q] = __fma_rn(ab, cv, -fx);
              t[rr][1][q] = -__fma_rn(ab, cu, yE[rr]);
              t[rr][2][q] = -(dx + yM[rr]) * rsg[rr][q];
            }
            if (N == 2 && i == 0) continue;
#pragma unroll
            for (int x = 0; x < 3; ++x) {
              double *out = reinterpret_cast<double *>(sm + S::OUT) + x * FE + at, base[N];
              lane_load<N>(out, base);
              if constexpr (S::ACC_IN || S::ACC_OUT) {
                double *ac = reinterpret_cast<double *>(sm + S::ACC) + x * FE + at, s[N];
                if constexpr (S::ACC_IN) lane_load<N>(ac, s);
                if constexpr (KIND == RK4_S1) lane_store<N>(ac, t[rr][x]);
                else {
#pragma unroll
                  for (int y = 0; y < N; ++y)
                    if constexpr (S::ACC_OUT) s[y] = __fma_rn(2., t[rr][x][y], s[y]);
                    else t[rr][x][y] = (s[y] + t[rr][x][y]) * (1. / 6.);
                  if constexpr (S::ACC_OUT) lane_store<N>(ac, s);
                }
              }
#pragma unroll
              for (int y = 0; y < N; ++y)
                base[y] = S::RK3 ? __fma_rn(KB, base[y], t[rr][x][y]) : __fma_rn(inc, t[rr][x][y], base[y]);
              lane_store<N>(out, base);
            }
          }
        }
      }
      if (c >= r0) {
        par1 ^= 1u;
        // ---- store the finished rows, one point per lane
        __syncwarp();
        const int lo = c == r0 ? H - 1 : 0, hi = (c == r1 && r1 < g.Nc) ? H - 1 : H;
        for (int rr = lo; rr < hi; ++rr) {
          const int gj = (c - 1) * H + 1 + rr;  // 0-based interior row
          const long long ro = fbase + (long long)(gj + H) * P + (X0 + H) + lane;
          double *const go[3] = {a.uo + ro, a.vo + ro, a.po + ro};
          const double *f = reinterpret_cast<const double *>(sm + S::OUT) + rr * RE + rem + H + lane;
#pragma unroll
          for (int kk = 0; kk < H; ++kk) {
            if (lane + 32 * kk < cnt) {
#pragma unroll
              for (int x = 0; x < 3; ++x) go[x][32 * kk] = f[x * FE + 32 * kk];
            }
          }
          if constexpr (S::ACC_OUT) {
            double *const ga[3] = {a.aU + ro, a.aV + ro, a.aP + ro};
            const double *fa = reinterpret_cast<const double *>(sm + S::ACC) + rr * RE + rem + H + lane;
#pragma unroll
            for (int kk = 0; kk < H; ++kk) {
              if (lane + 32 * kk < cnt) {
#pragma unroll
                for (int x = 0; x < 3; ++x) ga[x][32 * kk] = fa[x * FE + 32 * kk];
              }
            }
          }
          const int n = g.n;
          if (c0 == 0 || last_x || gj == 0 || gj == n - 1) {
            // pre-unification boundary values for the halo kernel
            double4 *bd = a.bnd + ((long long)mem * 6 + panel) * 4 * n;
            for (int t = lane; t < cnt; t += 32) {
              const int gi = c0 * H + t;
              const double *ft = f - lane + t;
              const double4 val = make_double4(ft[0], ft[FE], ft[2 * FE], 0.);
              if (gi == 0) bd[0 * n + gj] = val;
              if (gi == n - 1) bd[1 * n + gj] = val;
              if (gj == 0) bd[2 * n + gi] = val;
              if (gj == n - 1) bd[3 * n + gi] = val;
            }
          }
        }
        if (c < r1) {
          hand_to_copies();
          if (elect_one()) {
            issue_up(c);
          }
          __syncwarp();
        }
      }
      if (c < r1) {
        // ---- x sweep (:63-93) of the new rows (of the lower halo cell only the interface row is owned)
#pragma unroll
        for (int rr = 0; rr < H; ++rr) {
          if (c < r0 && rr < H - 1) continue;
          const Row &z = o[rr];
          double f[D], b1, b2;
          // ends of u (E's Riemann field), phiG and v; the point shared with the next cell by shuffle
          const double lamR = __shfl_down_sync(ALL, z.lx, 1);
#pragma unroll
          for (int i = 0; i < H; ++i) f[i] = z.u[i];
          f[H] = __shfl_down_sync(ALL, z.u[0], 1);
          const double lU = end_left<D>(f), rU_ = end_right<D>(f);
#pragma unroll
          for (int i = 0; i < H; ++i) f[i] = z.pg[i];
          f[H] = __shfl_down_sync(ALL, z.pg[0], 1);
          const double lQ = end_left<D>(f), rQ = end_right<D>(f);
          // E with Riemann on u
#pragma unroll
          for (int i = 0; i < H; ++i) f[i] = z.e[i];
          f[H] = __shfl_down_sync(ALL, z.e[0], 1);
          const double pE = __shfl_up_sync(ALL, __fma_rn(lamR, rU_, end_right<D>(f)), 1);
          const double gE = 0.5 * (pE + __fma_rn(-z.lx, lU, end_left<D>(f)));
          const double hE = __shfl_down_sync(ALL, gE, 1);
          interior64<D>(gE, f, b1, b2);
          double x[H];
          x[0] = gE;
          x[1] = interior64_end1<D>(b1, hE);
          if constexpr (D == 4) x[2] = interior64_end2(b2, hE);
#pragma unroll
          for (int i = 0; i < H; ++i) ar[(rr * H + i) * 32] = S::RK3 ? __fma_rn(KU, z.u[i], -inc * x[i]) : x[i];
          // phiG cU with Riemann on phiG
#pragma unroll
          for (int i = 0; i < H; ++i) f[i] = z.pg[i] * z.cu[i];
          f[H] = __shfl_down_sync(ALL, f[0], 1);
          const double pM = __shfl_up_sync(ALL, __fma_rn(lamR, rQ, end_right<D>(f)), 1);
          const double gM = 0.5 * (pM + __fma_rn(-z.lx, lQ, end_left<D>(f)));
          const double hM = __shfl_down_sync(ALL, gM, 1);
          interior64<D>(gM, f, b1, b2);
          x[0] = gM;
          x[1] = interior64_end1<D>(b1, hM);
          if constexpr (D == 4) x[2] = interior64_end2(b2, hM);
#pragma unroll
          for (int i = 0; i < H; ++i) ar[PE + (rr * H + i) * 32] = S::RK3 ? __fma_rn(KU, z.pg[i], -inc * x[i]) : x[i];
          // dvdx, upwinded by cU
#pragma unroll
          for (int i = 0; i < H; ++i) f[i] = z.v[i];
          f[H] = __shfl_down_sync(ALL, z.v[0], 1);
          const double pV = __shfl_up_sync(ALL, end_right<D>(f), 1);
          const double gV = z.cu[0] < 0. ? end_left<D>(f) : pV;
          const double hV = __shfl_down_sync(ALL, gV, 1);
          interior64<D>(gV, f, b1, b2);
          x[0] = gV;
          x[1] = interior64_end1<D>(b1, hV);
          if constexpr (D == 4) x[2] = interior64_end2(b2, hV);
#pragma unroll
          for (int i = 0; i < H; ++i) {
            ar[2 * PE + (rr * H + i) * 32] = x[i];
            ar[3 * PE + (rr * H + i) * 32] = z.cu[i];
            if constexpr (S::RK3) ar[4 * PE + (rr * H + i) * 32] = z.v[i];
          }
        }
        if (!wait_for(0, par0)) return;
        par0 ^= 1u;
      }
      __syncwarp();
    }
  }
  }
}

}  // namespace mcv
