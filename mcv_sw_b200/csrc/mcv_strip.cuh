// mcv_strip.cuh -- the stage kernel in strip form (split precision): one RK
// stage of MCV_SW (src/spatial_operators_mod.F90:12-133 fused with the stage
// update, src/time_scheme_mod.F90:71-123) with one warp per strip of cells.
//
// A warp owns up to 29 cells of a cell row and marches along y, one cell row
// per iteration; lane l holds the H x H points (H = D - 1) of cell column
// c0 - 1 + l, lanes 0 and w + 1 the halo cells.  Values of the neighbours in x
// come by shuffles, those in y stay in the lane's registers, so a cell row
// costs no block barrier and every point's quantities are formed once (the
// strip's two halo rows and columns apart).  The input rows of the next cell
// row and the operands of the next update are copied into shared memory (TMA)
// while this one is worked on; results leave through shared memory, so that
// the stores are coalesced although a lane holds H consecutive points.
//
// The fields of the momentum tendencies (E, u, v) are differenced in FP64 cell
// by cell: with the chord p0 -> pH of a cell's line, t = pH - p0, the one-sided
// derivatives are the chord's slope plus those of the residuals p_m - p0 -
// t m/H (zero at both ends), which are rounded to FP32; jumps between cells
// take the difference of the two chords in FP64.  phiG and its fluxes are
// rounded as they are, so that the fluxes of a seam agree bit for bit wherever
// they are formed and the flux form keeps conserving mass.
//
// A point's arithmetic does not depend on how the grid is cut into strips, and
// the file is compiled without FMA contraction, so that every instantiation
// gives the same bits.
#pragma once
#include "mcv_stage.cuh"

namespace mcv {


// one lane of the (converged) warp, which the compiler knows to be one
__device__ __forceinline__ bool elect_one() {
  uint32_t p;
  asm volatile(
      "{\n"
      " .reg .pred p;\n"
      " elect.sync _|p, 0xffffffff;\n"
      " selp.u32 %0, 1, 0, p;\n"
      "}\n"
      : "=r"(p));
  return p != 0;
}

// Before copies of an elected lane overwrite shared memory that the warp has used:
// every lane orders its own reads and writes before later ones of the async proxy
// (the fence acts on the accesses of the thread that executes it), then the warp
// meets.  One instruction for the warp, as the elected lane's alone would be.
__device__ __forceinline__ void hand_to_copies() {
  fence_proxy_async();
  __syncwarp();
}

// Shared memory of one warp for stage kind KIND: the staged input of a cell row
// ([field][H rows][RE] each), the operands and results of the update of the
// cell row before, the strip's metric entries in x, and the x sweep's results.
constexpr size_t align128(size_t x) { return (x + 127) / 128 * 128; }
template <int D, int KIND>
struct StripSmem {
  static constexpr int H = D - 1;
  static constexpr int RP = 32 * H;  // points of a warp's row
  static constexpr int RE = RP + 4;  // staged elements: a box starts at a multiple of 4 (16 bytes for either type)
  static constexpr bool FIRST = first_stage(KIND), LAST = last_stage(KIND);
  static constexpr bool RK3_INC = KIND == RK3_S2 || KIND == RK3_S3;                          // the update reads the input increment
  static constexpr bool ACC_IN = KIND == RK4_S2 || KIND == RK4_S3 || KIND == RK4_S4;        // ... the RK4 sum
  static constexpr bool ACC_OUT = KIND == RK4_S1 || KIND == RK4_S2 || KIND == RK4_S3;       // ... and writes it
  static constexpr int FB64 = (int)align128((size_t)H * RE * 8), FB32 = (int)align128((size_t)H * RE * 4);
  // The update's results take the place of what it last read: the last stage's
  // of Y + wd d (two slots of Y, the second filled by phase 0), RK3 stage 2's of d
  // (two slots of d); the others have an array of their own.
  static constexpr int NY = LAST ? 2 : 1, ND = FIRST ? 0 : (KIND == RK3_S2 ? 2 : 1);
  static constexpr int Y = 0, YS = 3 * FB64;               // Y_u, Y_v, Y_phi; a slot's size
  static constexpr int SG = Y + NY * YS;                   // sqrtG
  static constexpr int PS = SG + FB64;                     // phi_s
  static constexpr int DU = PS + FB32, DS = 3 * FB32;      // d_u, d_v, d_phi
  static constexpr int OUT = DU + ND * DS;                 // results, where not in place
  static constexpr int ACC = OUT + ((LAST || KIND == RK3_S2) ? 0 : DS);  // RK4 sums
  static constexpr int MET = ACC + ((ACC_IN || ACC_OUT) ? DS : 0);       // {1/sqrtG, sqrtG f} of the row to update
  static constexpr int MY = MET + FB64;                    // the rows' entries of the 1-D metric table
  static constexpr int XT = MY + 128;                      // {tan, cos^2/R^2} of the lane's columns: [2][RP] doubles
  static constexpr int AR = XT + 2 * RP * 8;               // x-sweep results: [H][H][32] float4, then [H][H][32] float
  static constexpr int FIRST_ROW = (int)(4 * RE * 8 + 4 * RE * 4 + 32);  // the strip's first row, staged over AR
  static constexpr int ARX = H * H * 32 * 20, ARB = (int)align128(ARX > FIRST_ROW ? ARX : FIRST_ROW);
  static constexpr int BAR = AR + ARB;
  static constexpr int BYTES = (int)align128(BAR + 16);
  // Warps per block, one block per SM: as many as registers (MCV4: 8) and shared
  // memory (227 KB) allow.  MCV3 takes 12, not the 16 that fit: with registers and
  // shared memory left over, blocks of the halo kernel become resident before the
  // strips end, and a stage with its halo kernel takes 26 us at Nc=181 instead of
  // 32, at no cost to large grids (64 members at Nc=128: 2.31 ms/step, was 2.40).
  static constexpr int WMAX = D == 3 ? 12 : 8;
  static constexpr int WPB = 232448 / BYTES < WMAX ? 232448 / BYTES : WMAX;
  static_assert(H * 32 <= 128, "metric entries of the rows");
};

// The quantities of one row of a lane's cell.
template <int H>
struct StripRow {
  double e[H], u[H], v[H];
  float pg[H], cu[H], cv[H];
  float lx;  // interface wave speed in x at the cell's first point
};

// All derivatives of the sweeps are per cell (times the cell width dx); the
// stage weights carry the 1/dx.
// One-sided derivatives of a line from its residuals r1, r2 over the chord
// (MCV4; MCV3 has r1 alone), without the chord's slope t.
template <int D>
__device__ __forceinline__ float chord_left(float r1, float r2) {
  if constexpr (D == 3) return 4.f * r1;
  else return fmaf(9.f, r1, -4.5f * r2);
}
template <int D>
__device__ __forceinline__ float chord_right(float r1, float r2) {
  if constexpr (D == 3) return -4.f * r1;
  else return fmaf(4.5f, r1, -9.f * r2);
}
// One-sided derivatives of a line from its points, two quantities at once
// (src/spatial_operators_mod.F90:204-238).
template <int D>
__device__ __forceinline__ float2 ends_left(const float2 *p) {
  if constexpr (D == 3) return fma2(bc2(-3.f), p[0], fma2(bc2(4.f), p[1], make_float2(-p[2].x, -p[2].y)));
  else return fma2(bc2(-5.5f), p[0], fma2(bc2(9.f), p[1], fma2(bc2(-4.5f), p[2], p[3])));
}
template <int D>
__device__ __forceinline__ float2 ends_right(const float2 *p) {
  if constexpr (D == 3) return fma2(bc2(3.f), p[2], fma2(bc2(-4.f), p[1], p[0]));
  else return fma2(bc2(5.5f), p[3], fma2(bc2(-9.f), p[2], fma2(bc2(4.5f), p[1], make_float2(-p[0].x, -p[0].y))));
}

// The chord of one line of a cell: t and the residuals.
template <int D>
__device__ __forceinline__ void chord(const double p0, const double p1, const double p2, const double pe, double &t,
                                      float &r1, float &r2) {
  t = pe - p0;
  if constexpr (D == 3) {
    r1 = (float)__fma_rn(-0.5, t, p1 - p0);
    r2 = 0.f;
  } else {
    r1 = (float)__fma_rn(-1. / 3., t, p1 - p0);
    r2 = (float)__fma_rn(-2. / 3., t, p2 - p0);
  }
}

// The interior points of a cell (src/spatial_operators_mod.F90:179-200) from
// its end derivatives: the part without the right end's.  Chord form: o0 is
// relative to the chord's slope, and so is the result.
template <int D>
__device__ __forceinline__ void interior_chord(float o0, float r1, float r2, float &b1, float &b2) {
  if constexpr (D == 3) {
    b1 = -0.25f * o0;
    b2 = 0.f;
  } else {
    const float k = r1 + r2;
    b1 = fmaf(-4.f / 27.f, o0, (2.f / 3.f) * k);
    b2 = fmaf(-5.f / 27.f, o0, (-2.f / 3.f) * k);
  }
}
template <int D>
__device__ __forceinline__ void interior_plain(float o0, const float *c, float &b1, float &b2) {
  const float via = c[D - 1] - c[0];
  if constexpr (D == 3) {
    b1 = fmaf(1.5f, via, -0.25f * o0);
    b2 = 0.f;
  } else {
    const float k = (2.f / 3.f) * ((c[0] + c[3]) - (c[1] + c[2]));
    b1 = fmaf(-4.f / 27.f, o0, fmaf(4.f / 3.f, via, -k));
    b2 = fmaf(-5.f / 27.f, o0, fmaf(4.f / 3.f, via, k));
  }
}
// ... and the right end's part
template <int D>
__device__ __forceinline__ float interior_end1(float b1, float o3) {
  return fmaf(D == 3 ? -0.25f : -5.f / 27.f, o3, b1);
}
__device__ __forceinline__ float interior_end2(float b2, float o3) { return fmaf(-4.f / 27.f, o3, b2); }

// A lane's H values of a shared-memory row.  MCV3: an even element (the rows, the
// strip's first point and the staged box all start at even ones), so that both
// points come in one access, without the two-way bank conflict of a stride of two.
// RK4 step of 16 members at Nc=128: 559 -> 538 us, FP64 735 -> 693.
template <int H, class T>
__device__ __forceinline__ void lane_load(const T *p, T (&o)[H]) {
  if constexpr (H == 2) {
    using V = std::conditional_t<sizeof(T) == 8, double2, float2>;
    const V v = *reinterpret_cast<const V *>(p);
    o[0] = v.x;
    o[1] = v.y;
  } else {
#pragma unroll
    for (int i = 0; i < H; ++i) o[i] = p[i];
  }
}
template <int H, class T>
__device__ __forceinline__ void lane_store(T *p, const T (&o)[H]) {
  if constexpr (H == 2) {
    using V = std::conditional_t<sizeof(T) == 8, double2, float2>;
    V v;
    v.x = o[0];
    v.y = o[1];
    *reinterpret_cast<V *>(p) = v;
  } else {
#pragma unroll
    for (int i = 0; i < H; ++i) p[i] = o[i];
  }
}

template <int D, int KIND, int NB, bool IDENT>
__global__ void __launch_bounds__(32 * StripSmem<D, KIND>::WPB, 1) strip_kernel(const __grid_constant__ StageBatch<NB> b) {
  using S = StripSmem<D, KIND>;
  constexpr int H = D - 1, RP = S::RP, RE = S::RE, WPB = S::WPB;
  constexpr unsigned ALL = 0xffffffffu;
  extern __shared__ __align__(128) unsigned char smraw[];
  const int lane = threadIdx.x & 31;
  const int warp = __shfl_sync(ALL, (int)(threadIdx.x >> 5), 0);  // uniform, and known to be
  unsigned char *sm = smraw + warp * S::BYTES;
  double *xt = reinterpret_cast<double *>(sm + S::XT);
  float4 *ar = reinterpret_cast<float4 *>(sm + S::AR) + lane;                    // x sweep: fx, dx, dvdx, cU
  float *arv = reinterpret_cast<float *>(sm + S::AR + H * H * 32 * 16) + lane;  // and cV of a point
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
    const long long fbase = (long long)mem * g.mstride + (long long)panel * g.plane;
    const int P = g.P;
    const float dx = (float)g.dx, wt = a.wt * (float)g.inv_dx;  // tendencies come times dx
    const float fdx = panel == 5 ? -dx : dx;
    if (id + stride >= b.total && x >= xe) allow_dependent_launch();
    // this lane's metric entries in x (lanes past the array: any valid one)
#pragma unroll
    for (int i = 0; i < H; ++i) {
      const double4 m = a.met1d[min(X0 + lane * H + i, g.np - 1)];
      xt[lane * H + i] = m.x;
      xt[RP + lane * H + i] = m.y;
    }
    const double r2 = a.r2;
    if (!waited) {
      wait_prerequisite_grid();  // the halo kernel before
      waited = true;
    }

    // ---- copies (lane 0).  Input of cell row c: padded rows (c + 1) H + 1 .. (c + 2) H.
    const int frow = (mem * 6 + panel) * g.np;
    constexpr uint32_t B64 = H * RE * 8, B32 = H * RE * 4;
    constexpr uint32_t IN_BYTES = 4 * B64 + B32 + (S::FIRST ? 0 : 3 * B32) + H * 32;
    // what the update before leaves alone: sqrtG, phi_s, the metric entries, and Y and d where
    // their slots are free
    auto issue_in1 = [&](int c) {
      const int row = (c + 1) * H + 1;
      tma_load_2d(sm + S::SG, &tm.f[3], X0a, row, bar);
      tma_load_2d(sm + S::PS, &tm.f[4], X0a, frow + row, bar);
      bulk_load(sm + S::MY, a.met1d + row, H * 32, bar);
      if constexpr (S::NY == 1) {
#pragma unroll
        for (int f = 0; f < 3; ++f) tma_load_2d(sm + S::Y + f * S::FB64, &tm.f[f], X0a, frow + row, bar);
      }
      if constexpr (S::ND == 1) {
#pragma unroll
        for (int f = 0; f < 3; ++f) tma_load_2d(sm + S::DU + f * S::FB32, &tm.f[5 + f], X0a, frow + row, bar);
      }
    };
    // what has two slots (RK3 stage 2: d; the last stage: Y), into the one whose results have left
    auto issue_in2 = [&](int c, int to) {
      const int row = (c + 1) * H + 1;
#pragma unroll
      for (int f = 0; f < 3; ++f) {
        if constexpr (S::ND == 2)
          tma_load_2d(sm + S::DU + to * S::DS + f * S::FB32, &tm.f[5 + f], X0a, frow + row, bar);
        if constexpr (S::NY == 2)
          tma_load_2d(sm + S::Y + to * S::YS + f * S::FB64, &tm.f[f], X0a, frow + row, bar);
      }
    };
    // operands of the update of cell row c's block
    constexpr uint32_t UP_BYTES = B64 + (S::ACC_IN ? 3 * B32 : 0);
    auto issue_up = [&](int c) {
      const int row = (c + 1) * H + 1;
      mbar_arrive_expect_tx(bar + 1, UP_BYTES);
      tma_load_2d(sm + S::MET, &tm.f[8], X0a, (panel < 4 ? 0 : g.np) + row, bar + 1);
      if constexpr (S::ACC_IN) {
#pragma unroll
        for (int f = 0; f < 3; ++f) tma_load_2d(sm + S::ACC + f * S::FB32, &tm.f[9 + f], X0a, frow + row, bar + 1);
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

    // pointwise quantities of one row (spatial_operators_mod.F90:58-61).  yf/sgf/psf/df: the row's
    // elements of lane 0 (Y fields fs apart, d fields ds apart); ly: the interface wave speeds in y
    // (for a row of interface points)
    auto row_values = [&](double *yf, int fs, const double *sgf, const float *psf, const float *df, int ds,
                          const double4 my, StripRow<H> &o, float *ly, bool base) {
      const double ty1 = __fma_rn(my.x, my.x, 1.), wy = (my.x * my.y) * r2;
      const int at = rem + lane * H;
      double y[3][H], sg[H], txs[H], cxs[H];
      float d[3][H], ps[H];
#pragma unroll
      for (int f = 0; f < 3; ++f) {
        lane_load<H>(yf + f * fs + at, y[f]);
        if constexpr (!S::FIRST) {
          lane_load<H>(df + f * ds + at, d[f]);
          if constexpr (KIND == RK3_S3) {
            // the update's base Y + wd d takes the place of these points' Y
            if (base) {
              double yb[H];
#pragma unroll
              for (int i = 0; i < H; ++i) yb[i] = __fma_rn((double)a.wd, (double)d[f][i], y[f][i]);
              lane_store<H>(yf + f * fs + at, yb);
            }
          }
        }
      }
      lane_load<H>(sgf + at, sg);
      lane_load<H>(psf + at, ps);
      lane_load<H>(xt + lane * H, txs);
      lane_load<H>(xt + RP + lane * H, cxs);
#pragma unroll
      for (int i = 0; i < H; ++i) {
        double u = y[0][i], v = y[1][i], p = y[2][i];
        if constexpr (!S::FIRST) {
          u += (double)d[0][i];
          v += (double)d[1][i];
          p += (double)d[2][i];
        }
        // equiangular metric from the 1-D tables (projection_mod.F90:150-192): rho2 = 1 + tan^2 x + tan^2 y,
        // G^11 = rho2 cx, G^22 = rho2 cy, G^12 = rho2 tan x cx tan y cy R^2 with c = cos^2/R^2
        const double tx = txs[i], cx = cxs[i];
        const double rho2 = __fma_rn(tx, tx, ty1), sxy = (tx * cx) * wy;
        const double cu = rho2 * __fma_rn(sxy, v, cx * u);  // cov2contrav, projection_mod.F90:138-148
        const double cv = rho2 * __fma_rn(sxy, u, my.y * v);
        o.u[i] = u;
        o.v[i] = v;
        // E = phi + phi_s + K (differenced below, so no mean depth is taken off)
        o.e[i] = __fma_rn(0.5, __fma_rn(cv, v, cu * u), p + (double)ps[i]);
        o.pg[i] = (float)(p * sg[i]);
        o.cu[i] = (float)cu;
        o.cv[i] = (float)cv;
        // max(|c - s|, |c + s|) = |c| + s, s = sqrt(G^ii phi) (:248-280)
        if (i == 0) {
          float r;
          asm("sqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"((float)(rho2 * cx) * (float)p));
          o.lx = fabsf(o.cu[0]) + r;
        }
        if (ly) {
          float r;
          asm("sqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"((float)(rho2 * my.y) * (float)p));
          ly[i] = fabsf(o.cv[i]) + r;
        }
      }
    };

    // ---- carried along y, per column of the lane: the last row's values and
    // the previous cell's chord, top-end derivatives and interior parts
    double e0[H], u0[H], v0[H];
    float m0[H], q0[H], lam0[H], cv0[H];
    double tE[H], tV[H];
    float sE[H], sU[H], rE[H], rV[H], rU[H], rM[H], rQ[H];
    float bE1[H], bE2[H], bM1[H], bM2[H], bU1[H], bU2[H];

    int sl = 0;  // the slot of the current cell row, where there are two
    hand_to_copies();
    if (elect_one()) {
      // the first row of the lower halo cell, then its block
      const int row = r0 * H, nel = min(RE, P - X0a);
      const long long o = fbase + (long long)row * P + X0a, om = (long long)row * P + X0a;
      unsigned char *fr = sm + S::AR;
      mbar_arrive_expect_tx(bar, IN_BYTES + (uint32_t)nel * (4 * 8 + 4 + (S::FIRST ? 0 : 12)) + 32);
      bulk_load(fr, a.yu + o, nel * 8, bar);
      bulk_load(fr + RE * 8, a.yv + o, nel * 8, bar);
      bulk_load(fr + 2 * RE * 8, a.yp + o, nel * 8, bar);
      bulk_load(fr + 3 * RE * 8, a.sgm + om, nel * 8, bar);
      bulk_load(fr + 4 * RE * 8, a.phis32 + o, nel * 4, bar);
      if constexpr (!S::FIRST) {
        bulk_load(fr + 4 * RE * 8 + RE * 4, a.du + o, nel * 4, bar);
        bulk_load(fr + 4 * RE * 8 + 2 * RE * 4, a.dv + o, nel * 4, bar);
        bulk_load(fr + 4 * RE * 8 + 3 * RE * 4, a.dp + o, nel * 4, bar);
      }
      bulk_load(fr + 4 * RE * 8 + 4 * RE * 4, a.met1d + row, 32, bar);
      issue_in1(r0 - 1);
      issue_in2(r0 - 1, 0);
      issue_up(r0 - 1);
    }
    __syncwarp();
    if (!wait_for(0, par0)) return;
    par0 ^= 1u;
    {
      StripRow<H> o;
      double *fr = reinterpret_cast<double *>(sm + S::AR);
      const float *fr32 = reinterpret_cast<const float *>(fr + 4 * RE);
      row_values(fr, RE, fr + 3 * RE, fr32, fr32 + RE, RE, *reinterpret_cast<const double4 *>(fr32 + 4 * RE), o,
                 nullptr, false);
#pragma unroll
      for (int i = 0; i < H; ++i) {
        e0[i] = o.e[i];
        u0[i] = o.u[i];
        v0[i] = o.v[i];
        q0[i] = o.pg[i];
        m0[i] = o.pg[i] * o.cv[i];
        lam0[i] = cv0[i] = 0.f;
        tE[i] = tV[i] = 0.;
        sE[i] = sU[i] = rE[i] = rV[i] = rU[i] = rM[i] = rQ[i] = 0.f;
        bE1[i] = bE2[i] = bM1[i] = bM2[i] = bU1[i] = bU2[i] = 0.f;
      }
    }
    const bool last_x = c0 + w == g.Nc;
    const int cnt = w * H + (last_x ? 1 : 0);  // owned points of a row

    for (int c = r0 - 1; c <= r1; ++c) {
      // ---- rows c H + 1 .. c H + H (interior indices) of the lane's cell
      StripRow<H> o[H];
      float ly[H];
      double *ycur = reinterpret_cast<double *>(sm + S::Y + (S::NY == 2 ? sl * S::YS : 0));
      const float *dcur = reinterpret_cast<const float *>(sm + S::DU + (S::ND == 2 ? sl * S::DS : 0));
#pragma unroll
      for (int rr = 0; rr < H; ++rr)
        row_values(ycur + rr * RE, S::FB64 / 8, reinterpret_cast<const double *>(sm + S::SG) + rr * RE,
                   reinterpret_cast<const float *>(sm + S::PS) + rr * RE, dcur + rr * RE, S::FB32 / 4,
                   reinterpret_cast<const double4 *>(sm + S::MY)[rr], o[rr], rr == H - 1 ? ly : nullptr, true);
      hand_to_copies();
      if (c < r1) {
        if (elect_one()) {
          mbar_arrive_expect_tx(bar, IN_BYTES);
          issue_in1(c + 1);
          if constexpr (S::ND == 2 || S::NY == 2) {
            // issue_in2 loads these when their slot is free, shortly before they are read
#pragma unroll
            for (int f = 0; f < 3; ++f)
              tma_prefetch_2d(&tm.f[S::ND == 2 ? 5 + f : f], X0a, frow + (c + 2) * H + 1);
          }
        }
        __syncwarp();
      }
      if (c >= r0)
        if (!wait_for(1, par1)) return;

      // ---- y sweep (:95-125) of the lane's columns: the fluxes at the bottom of
      // cell c, which complete rows (c - 1) H + 1 .. c H of cell c - 1; their
      // tendencies (:127-131) and RK stage update
      const float2 *met = reinterpret_cast<const float2 *>(sm + S::MET);
      float tt[H][3][H];                // tendencies of row, field, column
      [[maybe_unused]] float4 met2[H];  // MCV3: the entries of both columns
#pragma unroll
      for (int i = 0; i < H; ++i) {
        double t, tv, tu;
        float e1, e2, v1, v2, u1, u2;
        chord<D>(e0[i], o[0].e[i], o[1 % H].e[i], o[H - 1].e[i], t, e1, e2);
        chord<D>(v0[i], o[0].v[i], o[1 % H].v[i], o[H - 1].v[i], tv, v1, v2);
        chord<D>(u0[i], o[0].u[i], o[1 % H].u[i], o[H - 1].u[i], tu, u1, u2);
        const float slE = (float)t, slU = (float)tu;
        float fm[D], fq[D];
        fm[0] = m0[i];
        fq[0] = q0[i];
#pragma unroll
        for (int rr = 0; rr < H; ++rr) {
          fq[rr + 1] = o[rr].pg[i];
          fm[rr + 1] = o[rr].pg[i] * o[rr].cv[i];
        }
        float2 mq[D];
#pragma unroll
        for (int m = 0; m < D; ++m) mq[m] = make_float2(fm[m], fq[m]);
        const float2 lMQ = ends_left<D>(mq), rMQ = ends_right<D>(mq);
        const float lam = lam0[i];
        // E with Riemann on v, relative to this cell's chord
        const float dE = (float)(tE[i] - t), dV = (float)(tV[i] - tv);
        const float jump = (chord_left<D>(v1, v2) - rV[i]) - dV;
        const float gE = 0.5f * fmaf(-lam, jump, (rE[i] + chord_left<D>(e1, e2)) + dE);
        // phiG cV with Riemann on phiG
        const float gM = 0.5f * fmaf(-lam, lMQ.y - rQ[i], rM[i] + lMQ.x);
        // dudy, upwinded by cV (:83-85)
        const float lU = chord_left<D>(u1, u2);
        const bool down = cv0[i] < 0.f;
        const float gU = down ? slU + lU : sU[i] + rU[i];
        if (c >= r0) {
          const float o3 = gE - dE, u3 = down ? lU - (sU[i] - slU) : rU[i];  // relative to cell c - 1's chord
          float fy[H], dy[H], dudy[H];
          fy[0] = sE[i] + interior_end1<D>(bE1[i], o3);
          dy[0] = interior_end1<D>(bM1[i], gM);
          dudy[0] = sU[i] + interior_end1<D>(bU1[i], u3);
          if constexpr (D == 4) {
            fy[1] = sE[i] + interior_end2(bE2[i], o3);
            dy[1] = interior_end2(bM2[i], gM);
            dudy[1] = sU[i] + interior_end2(bU2[i], u3);
          }
          fy[H - 1] = slE + gE;
          dy[H - 1] = gM;
          dudy[H - 1] = gU;
          // MCV4: the column's operands before its first result is stored, past which the compiler moves no
          // load (RK4 step at Nc=512 1016 -> 943 us, RK3 at Nc=256 199 -> 192; MCV3 has no registers for it)
          [[maybe_unused]] float4 xs[H];
          [[maybe_unused]] float cvs[H], up[H][3];  // up: RK4 sum or (RK3 stage 2) d
          [[maybe_unused]] float2 ms[H];
          if constexpr (H == 3) {
#pragma unroll
            for (int rr = 0; rr < H; ++rr) {
              const int at = rr * RE + rem + lane * H + i;
              xs[rr] = ar[(rr * H + i) * 32];
              cvs[rr] = arv[(rr * H + i) * 32];
              ms[rr] = met[at];
#pragma unroll
              for (int f = 0; f < 3; ++f) {
                if constexpr (S::ACC_IN) up[rr][f] = reinterpret_cast<const float *>(sm + S::ACC + f * S::FB32)[at];
                if constexpr (KIND == RK3_S2)
                  up[rr][f] = reinterpret_cast<const float *>(sm + S::DU + (sl ^ 1) * S::DS + f * S::FB32)[at];
              }
            }
          }
#pragma unroll
          for (int rr = 0; rr < H; ++rr) {
            const int at = rr * RE + rem + lane * H;
            const float4 x = H == 3 ? xs[rr] : ar[(rr * H + i) * 32];  // fx, dx, dvdx, cU
            const float cv = H == 3 ? cvs[rr] : arv[(rr * H + i) * 32];
            float2 m;  // 1/sqrtG, sqrtG f
            if constexpr (H == 2) {
              if (i == 0) met2[rr] = *reinterpret_cast<const float4 *>(met + at);
              m = i == 0 ? make_float2(met2[rr].x, met2[rr].y) : make_float2(met2[rr].z, met2[rr].w);
            } else {
              m = ms[rr];
            }
            // sqrtG (vort + f) = (dvdx - dudy) + sqrtG f
            const float ab = fmaf(fdx, m.y, x.z - dudy[rr]);
            // tendencies of u, v, phi (that of phiG over sqrtG)
            tt[rr][0][i] = fmaf(ab, cv, -x.x);
            tt[rr][1][i] = fmaf(-ab, x.w, -fy[rr]);
            tt[rr][2][i] = -(x.y + dy[rr]) * m.x;
            // the update: MCV4 point by point, MCV3 both points of the lane at once
            constexpr int N = H == 2 ? 2 : 1;
            if (N == 2 && i == 0) continue;
            const int at0 = at + (N == 2 ? 0 : i);
#pragma unroll
            for (int f = 0; f < 3; ++f) {
              float sum[N];
#pragma unroll
              for (int q = 0; q < N; ++q) sum[q] = tt[rr][f][N == 2 ? q : i];
              if constexpr (S::ACC_IN || S::ACC_OUT) {
                float *pa = reinterpret_cast<float *>(sm + S::ACC + f * S::FB32) + at0;
                float ac[N];
                if constexpr (S::ACC_IN && H == 3) ac[0] = up[rr][f];
                else if constexpr (S::ACC_IN) lane_load<N>(pa, ac);
                if constexpr (KIND == RK4_S1) lane_store<N>(pa, sum);
                else {
#pragma unroll
                  for (int q = 0; q < N; ++q)
                    if constexpr (S::ACC_OUT) ac[q] = fmaf(2.f, sum[q], ac[q]);
                    else sum[q] = (ac[q] + sum[q]) * (1.f / 6.f);
                  if constexpr (S::ACC_OUT) lane_store<N>(pa, ac);
                }
              }
              if constexpr (S::LAST) {
                double *py = reinterpret_cast<double *>(sm + S::Y + (sl ^ 1) * S::YS + f * S::FB64) + at0;
                double y[N];
                lane_load<N>(py, y);
#pragma unroll
                for (int q = 0; q < N; ++q) y[q] = y[q] + (double)(wt * sum[q]);
                lane_store<N>(py, y);
              } else if constexpr (KIND == RK3_S2) {
                float *pd = reinterpret_cast<float *>(sm + S::DU + (sl ^ 1) * S::DS + f * S::FB32) + at0;
                float d[N];
                if constexpr (H == 3) d[0] = up[rr][f];
                else lane_load<N>(pd, d);
#pragma unroll
                for (int q = 0; q < N; ++q) d[q] = fmaf(wt, sum[q], a.wd * d[q]);
                lane_store<N>(pd, d);
              } else {
                float r[N];
#pragma unroll
                for (int q = 0; q < N; ++q) r[q] = wt * sum[q];
                lane_store<N>(reinterpret_cast<float *>(sm + S::OUT + f * S::FB32) + at0, r);
              }
            }
          }
        }
        interior_chord<D>(gE, e1, e2, bE1[i], bE2[i]);
        interior_plain<D>(gM, fm, bM1[i], bM2[i]);
        interior_chord<D>(gU - slU, u1, u2, bU1[i], bU2[i]);
        tE[i] = t;
        tV[i] = tv;
        sE[i] = slE;
        sU[i] = slU;
        rE[i] = chord_right<D>(e1, e2);
        rV[i] = chord_right<D>(v1, v2);
        rU[i] = chord_right<D>(u1, u2);
        rM[i] = rMQ.x;
        rQ[i] = rMQ.y;
        e0[i] = o[H - 1].e[i];
        u0[i] = o[H - 1].u[i];
        v0[i] = o[H - 1].v[i];
        q0[i] = fq[H];
        m0[i] = fm[H];
        lam0[i] = ly[i];
        cv0[i] = o[H - 1].cv[i];
      }

      if (c >= r0) {
        par1 ^= 1u;
        // ---- store the finished rows, one point per lane
        __syncwarp();
        const int lo = c == r0 ? H - 1 : 0, hi = (c == r1 && r1 < g.Nc) ? H - 1 : H;
        using Out = std::conditional_t<S::LAST, double, float>;
        constexpr int FB = S::LAST ? S::FB64 : S::FB32;
        const Out *res = reinterpret_cast<const Out *>(
            sm + (S::LAST ? S::Y + (sl ^ 1) * S::YS : KIND == RK3_S2 ? S::DU + (sl ^ 1) * S::DS : S::OUT));
        for (int rr = lo; rr < hi; ++rr) {
          const int gj = (c - 1) * H + 1 + rr;  // 0-based interior row
          const long long ro = fbase + (long long)(gj + H) * P + (X0 + H) + lane;
          Out *const go[3] = {(Out *)(S::LAST ? (void *)a.uo : (void *)a.eu) + ro,
                              (Out *)(S::LAST ? (void *)a.vo : (void *)a.ev) + ro,
                              (Out *)(S::LAST ? (void *)a.po : (void *)a.ep) + ro};
          const Out *f = res + rr * RE + rem + H + lane;
#pragma unroll
          for (int kk = 0; kk < H; ++kk) {
            if (lane + 32 * kk < cnt) {
#pragma unroll
              for (int x = 0; x < 3; ++x) go[x][32 * kk] = f[x * (FB / (int)sizeof(Out)) + 32 * kk];
            }
          }
          if constexpr (S::ACC_OUT) {
            float *const ga[3] = {a.fU + ro, a.fV + ro, a.fP + ro};
            const float *fa = reinterpret_cast<const float *>(sm + S::ACC) + rr * RE + rem + H + lane;
#pragma unroll
            for (int kk = 0; kk < H; ++kk) {
              if (lane + 32 * kk < cnt) {
#pragma unroll
                for (int x = 0; x < 3; ++x) ga[x][32 * kk] = fa[x * (S::FB32 / 4) + 32 * kk];
              }
            }
          }
          const int n = g.n;
          if (c0 == 0 || last_x || gj == 0 || gj == n - 1) {
            // pre-unification boundary values for the halo kernel
            const long long bo = ((long long)mem * 6 + panel) * 4 * n;
            for (int t = lane; t < cnt; t += 32) {
              const int gi = c0 * H + t;
              const Out *ft = res + rr * RE + rem + H + t;
              const Out v0_ = ft[0], v1_ = ft[FB / (int)sizeof(Out)], v2_ = ft[2 * (FB / (int)sizeof(Out))];
              auto put = [&](int at) {
                if constexpr (S::LAST) a.bnd[bo + at] = make_double4(v0_, v1_, v2_, 0.);
                else a.bnd32[bo + at] = make_float4(v0_, v1_, v2_, 0.f);
              };
              if (gi == 0) put(0 * n + gj);
              if (gi == n - 1) put(1 * n + gj);
              if (gj == 0) put(2 * n + gi);
              if (gj == n - 1) put(3 * n + gi);
            }
          }
        }
      }
      if (c < r1) {
        hand_to_copies();
        if (elect_one()) {
          issue_in2(c + 1, sl ^ 1);
          if (c >= r0) issue_up(c);
        }
        __syncwarp();
      }
      sl ^= 1;
      if (c < r1) {
        // ---- x sweep (:63-93) of the new rows (of the lower halo cell only the
        // interface row is owned)
        auto sweep_row = [&](int rr) {
          const StripRow<H> &z = o[rr];
          float fm[D], fq[D];
#pragma unroll
          for (int i = 0; i < H; ++i) {
            fq[i] = z.pg[i];
            fm[i] = z.pg[i] * z.cu[i];
          }
          // the point shared with the next cell
          const double ee = __shfl_down_sync(ALL, z.e[0], 1), ue = __shfl_down_sync(ALL, z.u[0], 1),
                       ve = __shfl_down_sync(ALL, z.v[0], 1);
          fq[H] = __shfl_down_sync(ALL, fq[0], 1);
          fm[H] = __shfl_down_sync(ALL, fm[0], 1);
          double t, tu, tv;
          float e1, e2, v1, v2, u1, u2;
          chord<D>(z.e[0], z.e[1], z.e[2 % H], ee, t, e1, e2);
          chord<D>(z.u[0], z.u[1], z.u[2 % H], ue, tu, u1, u2);
          chord<D>(z.v[0], z.v[1], z.v[2 % H], ve, tv, v1, v2);
          const float slE = (float)t, slV = (float)tv;
          float2 mq[D];
#pragma unroll
          for (int m = 0; m < D; ++m) mq[m] = make_float2(fm[m], fq[m]);
          const float2 lMQ = ends_left<D>(mq), rMQ = ends_right<D>(mq);
          // the left neighbour's right end
          const double tp = __shfl_up_sync(ALL, t, 1), tup = __shfl_up_sync(ALL, tu, 1);
          const float pE = __shfl_up_sync(ALL, chord_right<D>(e1, e2), 1);
          const float pU = __shfl_up_sync(ALL, chord_right<D>(u1, u2), 1);
          const float pV = __shfl_up_sync(ALL, slV + chord_right<D>(v1, v2), 1);
          const float pM = __shfl_up_sync(ALL, rMQ.x, 1), pQ = __shfl_up_sync(ALL, rMQ.y, 1);
          const float dE = (float)(tp - t), dU = (float)(tup - tu);
          const float jump = (chord_left<D>(u1, u2) - pU) - dU;
          const float gE = 0.5f * fmaf(-z.lx, jump, (pE + chord_left<D>(e1, e2)) + dE);
          const float gM = 0.5f * fmaf(-z.lx, lMQ.y - pQ, pM + lMQ.x);
          const float gV = z.cu[0] < 0.f ? slV + chord_left<D>(v1, v2) : pV;
          // the fluxes at the cell's right end, relative to its chord
          const float hE = __shfl_down_sync(ALL, gE - dE, 1), hM = __shfl_down_sync(ALL, gM, 1),
                      hV = __shfl_down_sync(ALL, gV, 1) - slV;
          float b1, b2, d1, d2, w1, w2;
          interior_chord<D>(gE, e1, e2, b1, b2);
          interior_plain<D>(gM, fm, d1, d2);
          interior_chord<D>(gV - slV, v1, v2, w1, w2);
          float fx[H], dd[H], vx[H];
          fx[0] = slE + gE;
          dd[0] = gM;
          vx[0] = gV;
          fx[1] = slE + interior_end1<D>(b1, hE);
          dd[1] = interior_end1<D>(d1, hM);
          vx[1] = slV + interior_end1<D>(w1, hV);
          if constexpr (D == 4) {
            fx[2] = slE + interior_end2(b2, hE);
            dd[2] = interior_end2(d2, hM);
            vx[2] = slV + interior_end2(w2, hV);
          }
#pragma unroll
          for (int i = 0; i < H; ++i) {
            ar[(rr * H + i) * 32] = make_float4(fx[i], dd[i], vx[i], z.cu[i]);
            arv[(rr * H + i) * 32] = z.cv[i];
          }
        };
#pragma unroll
        for (int rr = 0; rr < H; ++rr)
          if (c >= r0 || rr == H - 1) sweep_row(rr);
        if (!wait_for(0, par0)) return;
        par0 ^= 1u;
      }
      __syncwarp();
    }
  }
  }
}

}  // namespace mcv
