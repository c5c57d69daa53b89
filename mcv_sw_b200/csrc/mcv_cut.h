// mcv_cut.h -- how a strip-form launch is divided between its warps: the cut, made
// on the host, and what a warp of mcv_strip.cuh / mcv_strip64.cuh takes of it.
// Plain C++ for the host, and device code under nvcc.
//
// B is a StageBatch, of which this uses, per grid k: g[k].Nc, g[k].n, slots[k]
// (active members) and the cut itself.  nsx columns of at most kStripCells cells lie
// across a panel.  Either (sy > 0) the columns of the first pm1 panels (of all
// members) are cut into sy segments of cell rows, those of the others into sy2,
// total strips in all, the first of a grid t0; or `total` runs of equal length share
// the columns of every grid laid end to end, kStripUnit units a cell row and
// kStripStart in front of each column, from unit t0 of a grid on: run id starts at
// id run_q + id run_r / total.
#pragma once
#include <algorithm>
#include <climits>
#include <cmath>

#ifdef __CUDACC__
#define MCV_CUT_FN __device__ __forceinline__
#else
#define MCV_CUT_FN inline
#endif

namespace mcv {

// owned cells per strip, lanes 1..29 (lane 31 lends its first point to lane 30)
constexpr int kStripCells = 29;
// What a strip pays for its start and its two halo rows, in cell rows: 2.25
// (measured: MCV4 Nc=256 stages fit (rows + 2.2) x 3.6 us split precision)
constexpr int kStripUnit = 8, kStripStart = 18;

// A strip: cells [c0, c0 + w) of cell rows [r0, r1) of one panel of one active
// member.  A warp takes, one after the other,
//  - segments of columns, cut alike over many panels: neighbouring columns are
//    worked on at the same rows at the same time, so that a row of a field is read
//    as a whole (panels fastest: split precision's six panels share the metric
//    planes); or
//  - a run of the columns laid end to end: the end of a column and the beginning
//    of another, so that no warp is left over.
struct Strip {
  int c0, w, r0, r1, panel, slot;
};
template <class B>
MCV_CUT_FN void strip_column(const B &b, int k, int pm, int col, Strip &t) {
  const int Nc = b.g[k].Nc, nsx = b.nsx[k];
  t.slot = pm / 6;
  t.panel = pm - 6 * t.slot;
  t.c0 = Nc * col / nsx;
  t.w = Nc * (col + 1) / nsx - t.c0;
}
// The work of item id is [x, xe): units of a run; segments are one each.
template <class B>
MCV_CUT_FN void strip_work(const B &b, int id, int &x, int &xe) {
  x = id * b.run_q + (int)((long long)id * b.run_r / b.total);
  xe = (id + 1) * b.run_q + (int)((long long)(id + 1) * b.run_r / b.total);
}
// The next strip of the warp whose work is item id, [x, xe) of it left (grid k);
// x moves past it.  False if the run holds no cell row of that column.
template <class B>
MCV_CUT_FN bool next_strip(const B &b, int id, int &x, int xe, int &k, Strip &t) {
  const bool segments = b.sy[0] > 0;
  const int at = segments ? id : x;
  k = 0;
#ifdef __CUDACC__
#pragma unroll
#endif
  for (int j = 1; j < B::kGrids; ++j)
    if (j < b.ngrids && at >= b.t0[j]) k = j;
  const int Nc = b.g[k].Nc, nsx = b.nsx[k];
  if (segments) {
    int local = id - b.t0[k], pm = 0, per = b.pm1[k], sy = b.sy[k];
    const int first = per * nsx * sy;
    if (local >= first) {
      local -= first;
      pm = per;
      per = 6 * b.slots[k] - per;
      sy = b.sy2[k];
    }
    const int q = local / per, seg = q / nsx;
    strip_column(b, k, pm + local - q * per, q - seg * nsx, t);
    t.r0 = Nc * seg / sy;
    t.r1 = Nc * (seg + 1) / sy;
    x = xe;
    return true;
  }
  const int len = Nc * kStripUnit + kStripStart;
  const int column = (x - b.t0[k]) / len, start = b.t0[k] + column * len, pm = column / nsx;
  strip_column(b, k, pm, column - pm * nsx, t);
  auto row = [&](int y) {
    const int u = y - start - kStripStart + kStripUnit / 2;
    return (u > 0 ? u : 0) / kStripUnit;
  };
  t.r0 = row(x);
  x = xe < start + len ? xe : start + len;
  t.r1 = row(x);
  return t.r1 > t.r0;
}

// Divides the columns of a strip-form launch over b's first n grids between
// `warps` resident warps (StageBatch, mcv_strip.cuh).  The cost of a cut is that of
// its longest warp, in cell rows, a strip paying kStart for its start and halo rows.
//  - Segments of about the same number of cell rows in every column, as many as
//    cost least.
//  - Segments of two lengths, where that costs 5% less and there are several
//    members: whole passes of long segments for some of the panels, then short ones
//    for the others.  64 members of MCV3 Nc=128 take whole columns for 355 panels
//    and twelfths for 29 instead of 16ths for all: RK4 2.37 -> 2.19 ms/step split
//    precision; 50 of Nc=100 FP64 1.51 -> 1.32.  Where less is promised or panels
//    are few and large it was lost (MCV4 Nc=700 FP64: 2.98 -> 3.16).
//  - One run per warp, where that costs 4% less and neighbouring columns stay in
//    step: they share sectors at their seams, which are read twice where the
//    neighbour's are no longer in L2.  What a stage touches (76 bytes a point, FP64
//    130) stays there up to 126 MB (4 members of MCV3 Nc=128 split precision: RK4
//    180 -> 169 us).  Other grids want a column to be a whole number of runs (MCV4
//    Nc=256 FP64, 10.96: RK3 283 -> 276 us; Nc=280, 9.87: RK4 551 -> 596; 4 members
//    of MCV3 Nc=181 split precision, 10.57: 275 -> 306) and runs to be short (MCV3
//    Nc=512 FP64, 47 rows, 10.96: 738 -> 827).  Few points, and the rule gives
//    up the runs of 8 members of MCV4 Nc=96 split precision, which were 1% faster
//    (450 us; segments 456).
// bytes: what a stage touches per point (76 split precision, 130 FP64).  False: too
// many cell rows to number.
template <class B>
inline bool cut_strips(B &b, int n, int warps, int bytes) {
  constexpr double kStart = (double)kStripStart / kStripUnit;
  constexpr long long kLongRun = 32;  // cell rows
  long long units = 0, rows = 0, points = 0;
  int most = 1;
  for (int k = 0; k < n; ++k) {
    b.nsx[k] = (b.g[k].Nc + kStripCells - 1) / kStripCells;
    const long long columns = 6LL * b.slots[k] * b.nsx[k];
    units += columns * (b.g[k].Nc * kStripUnit + kStripStart);
    rows += columns * b.g[k].Nc;
    points += 6LL * b.slots[k] * b.g[k].n * b.g[k].n;
    most = std::max(most, b.g[k].Nc);
  }
  if (units > INT_MAX / 2) return false;
  double best = 1e300;
  int len = 1;
  for (int l = 1; l <= most; ++l) {
    long long strips = 0;
    for (int k = 0; k < n; ++k) strips += 6LL * b.slots[k] * b.nsx[k] * ((b.g[k].Nc + l - 1) / l);
    const double cost = (double)((strips + warps - 1) / warps) * (l + kStart);
    if (cost < best) {
      best = cost;
      len = l;
    }
  }
  int pm1 = 0, sy1 = 0, sy2 = 0;
  if (n == 1 && b.slots[0] > 1) {
    const int Nc = b.g[0].Nc, nsx = b.nsx[0], per = 6 * b.slots[0];
    double split = 0.95 * best;
    for (int s1 = 1; s1 <= Nc; ++s1) {
      const long long strip = (long long)nsx * s1;  // strips of a panel
      const int passes = (int)(per * strip / warps), m = (int)((long long)passes * warps / strip);
      if (m <= 0 || m >= per) continue;
      const double long1 = passes * ((Nc + s1 - 1) / s1 + kStart);
      if (long1 >= split) continue;
      for (int p2 = 1; p2 <= 3; ++p2) {
        const int s2 = (int)std::min<long long>(Nc, (long long)p2 * warps / ((long long)(per - m) * nsx));
        if (s2 < 1) continue;
        const double cost = long1 + p2 * ((Nc + s2 - 1) / s2 + kStart);
        if (cost < split) {
          split = cost;
          pm1 = m;
          sy1 = s1;
          sy2 = s2;
        }
      }
    }
    if (pm1) best = split;
  }
  const long long run = (units + (long long)warps * kStripUnit - 1) / ((long long)warps * kStripUnit);  // cell rows, up
  bool runs = run <= kLongRun && (double)run + kStart < 0.96 * best;
  const bool cached = points * bytes <= (126ll << 20);
  for (int k = 0; k < n && !cached; ++k) {
    const double per_column = (double)(b.g[k].Nc * kStripUnit + kStripStart) * warps / (double)units;
    runs = runs && std::abs(per_column - std::round(per_column)) <= 0.1;
  }
  b.ngrids = n;
  int at = 0;
  for (int k = 0; k < n; ++k) {
    const int columns = 6 * b.slots[k] * b.nsx[k];
    b.t0[k] = at;
    b.pm1[k] = pm1 ? pm1 : 6 * b.slots[k];
    b.sy[k] = runs ? 0 : pm1 ? sy1 : (b.g[k].Nc + len - 1) / len;
    b.sy2[k] = sy2;
    at += runs ? columns * (b.g[k].Nc * kStripUnit + kStripStart)
               : b.pm1[k] * b.nsx[k] * b.sy[k] + (6 * b.slots[k] - b.pm1[k]) * b.nsx[k] * sy2;
  }
  b.t0[n] = at;
  b.total = runs ? (int)std::min<long long>(warps, rows) : at;
  b.run_q = at / b.total;
  b.run_r = at % b.total;
  return true;
}

}  // namespace mcv
