// The cut of a strip-form launch (mcv_cut.h), walked as the kernels walk it: every
// cell of every panel of every member in exactly one strip, strips within their
// limits, and the forms that the cut can take all seen.
//
//   cut_test            checks random launches and the listed ones, prints "ok"
//   cut_test warps bytes nc:members ...   prints what one launch's cut is
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <random>
#include <vector>

#include "mcv_cut.h"

namespace {

struct Grid {
  int Nc, n;
};
template <int NB>
struct Batch {
  static constexpr int kGrids = NB;
  Grid g[NB];
  int ngrids, total, slots[NB];
  int nsx[NB], sy[NB], sy2[NB], pm1[NB], t0[NB + 1];
  int run_q, run_r;
};

struct Kind {
  bool runs = false, two_lengths = false, several = false, column_end = false, grid_end = false;
};

#define REQUIRE(cond)                                                    \
  if (!(cond)) {                                                         \
    std::printf("line %d: %s (%s)\n", __LINE__, #cond, what);            \
    std::exit(1);                                                        \
  }

template <int NB>
Kind check(int order, const std::vector<std::pair<int, int>> &grids, int blocks_limit, int wpb, int bytes) {
  char what[256];
  int at = std::snprintf(what, sizeof what, "order %d, %d x %d warps, %d bytes", order, blocks_limit, wpb, bytes);
  Batch<NB> b;
  std::memset(&b, 0, sizeof b);
  const int n = (int)grids.size();
  for (int k = 0; k < n; ++k) {
    b.g[k] = Grid{grids[k].first, grids[k].first * (order - 1) + 1};
    b.slots[k] = grids[k].second;
    if (at < 200) at += std::snprintf(what + at, sizeof what - at, ", %d:%d", grids[k].first, grids[k].second);
  }
  REQUIRE(mcv::cut_strips(b, n, blocks_limit * wpb, bytes));
  REQUIRE(b.total > 0 && b.ngrids == n);
  const int blocks = std::max(1, std::min(b.total, blocks_limit));
  std::vector<std::vector<unsigned char>> seen(n);
  for (int k = 0; k < n; ++k) seen[k].assign((size_t)6 * b.slots[k] * b.g[k].Nc * b.g[k].Nc, 0);
  Kind kind;
  kind.runs = b.sy[0] == 0;
  kind.two_lengths = !kind.runs && b.pm1[0] < 6 * b.slots[0];
  for (int block = 0; block < blocks; ++block)
    for (int warp = 0; warp < wpb; ++warp) {
      int strips = 0;
      for (int id = warp * blocks + block; id < b.total; id += blocks * wpb) {
        int x, xe, last = -1;
        mcv::strip_work(b, id, x, xe);
        REQUIRE(x >= 0 && xe > x && xe <= (kind.runs ? b.t0[n] : b.total));
        int columns = 0;
        while (x < xe) {
          const int before = x;
          int k;
          mcv::Strip s;
          const bool any = mcv::next_strip(b, id, x, xe, k, s);
          REQUIRE(x > before && x <= xe);
          REQUIRE(k >= 0 && k < n);
          if (!any) continue;
          const int Nc = b.g[k].Nc;
          REQUIRE(s.slot >= 0 && s.slot < b.slots[k] && s.panel >= 0 && s.panel < 6);
          REQUIRE(s.w >= 1 && s.w <= mcv::kStripCells && s.c0 >= 0 && s.c0 + s.w <= Nc);
          REQUIRE(s.r0 >= 0 && s.r1 > s.r0 && s.r1 <= Nc);
          for (int r = s.r0; r < s.r1; ++r)
            for (int c = s.c0; c < s.c0 + s.w; ++c) {
              unsigned char &cell = seen[k][(((size_t)s.slot * 6 + s.panel) * Nc + r) * Nc + c];
              REQUIRE(cell == 0);
              cell = 1;
            }
          ++strips;
          kind.column_end |= ++columns > 1;
          kind.grid_end |= last >= 0 && last != k;
          last = k;
        }
      }
      kind.several |= strips > 1;
    }
  for (int k = 0; k < n; ++k)
    for (unsigned char cell : seen[k]) REQUIRE(cell == 1);
  return kind;
}

Kind check_any(int order, const std::vector<std::pair<int, int>> &grids, int blocks, int wpb, int bytes) {
  return grids.size() == 1 ? check<1>(order, grids, blocks, wpb, bytes) : check<4>(order, grids, blocks, wpb, bytes);
}

}  // namespace

int main(int argc, char **argv) {
  if (argc > 3) {
    std::vector<std::pair<int, int>> grids;
    for (int i = 3; i < argc; ++i) {
      int nc = 0, m = 1;
      std::sscanf(argv[i], "%d:%d", &nc, &m);
      grids.push_back({nc, m});
    }
    const Kind k = check_any(4, grids, 148, std::atoi(argv[1]), std::atoi(argv[2]));
    std::printf("runs %d two_lengths %d several %d column_end %d grid_end %d\n", k.runs, k.two_lengths, k.several,
                k.column_end, k.grid_end);
    return 0;
  }
  // warps per block and bytes of the forms that exist: FP64 MCV3, MCV4, split precision MCV3, MCV4
  const int forms[][3] = {{3, 8, 130}, {3, 6, 130}, {4, 4, 130}, {3, 12, 76}, {3, 10, 76}, {4, 8, 76}, {4, 7, 76}, {4, 6, 76}};
  std::mt19937 rng(7);
  auto uniform = [&](int a, int b) { return a + (int)(rng() % (unsigned)(b - a + 1)); };
  bool runs = false, runs_over_grids = false, two = false, several = false, several_grids = false;
  auto note = [&](const Kind &k, size_t n) {
    runs |= k.runs && k.column_end;
    runs_over_grids |= k.runs && k.grid_end;
    two |= k.two_lengths;
    several |= !k.runs && k.several && n == 1;
    several_grids |= !k.runs && k.several && n > 1;
  };
  for (const auto &f : forms) {
    for (int nc = 2; nc <= 130; ++nc) note(check_any(f[0], {{nc, 1}}, 148, f[1], f[2]), 1);
    for (int nc : {134, 161, 181, 256, 280, 512}) note(check_any(f[0], {{nc, 1}}, 148, f[1], f[2]), 1);
    for (int it = 0; it < 150; ++it) {
      const int n = uniform(1, 4);
      std::vector<std::pair<int, int>> grids;
      for (int k = 0; k < n; ++k) {
        const int nc = uniform(2, it % 3 ? 130 : 40);
        grids.push_back({nc, uniform(1, std::max(1, 300000 / (nc * nc * 6 * n)) > 60 ? 60 : std::max(1, 300000 / (nc * nc * 6 * n)))});
      }
      note(check_any(f[0], grids, uniform(0, 3) ? 148 : uniform(1, 40), f[1], f[2]), grids.size());
    }
  }
  if (!(runs && runs_over_grids && two && several && several_grids)) {
    std::printf("not seen: runs %d over grids %d two lengths %d several %d, of grids %d\n", runs, runs_over_grids, two,
                several, several_grids);
    return 1;
  }
  std::printf("ok\n");
  return 0;
}
