// Shares the tiles of random products out and checks that every tile is somebody's, once, and that the units'
// loads are what handing the tiles out one by one, longest first, gives.  Arguments: seed, trials.
#include <cstdio>
#include <cstdlib>
#include <queue>
#include <random>
#include <vector>

#include "zp_share.cuh"

int main(int argc, char **argv) {
  std::mt19937 rng(std::atoi(argv[1]));
  auto pick = [&](int lo, int hi) { return std::uniform_int_distribution<int>(lo, hi)(rng); };
  for (int trial = 0; trial < std::atoi(argv[2]); ++trial) {
    const int n = pick(1, ZP_GEMM_GROUP), units = pick(0, 1) ? 148 : pick(1, 80);
    GroupPlan pl;
    for (int k = 0; k < n; ++k) {
      pl.shape[k].tiles = pick(0, 2) ? pick(1, 3000) : pick(0, 60);
      pl.shape[k].cost = pick(0, 3) ? pick(500, 60000) : 4000;      // equal ones among them
    }
    std::sort(pl.shape, pl.shape + n, [](const Shape &a, const Shape &b) { return a.cost > b.cost; });
    share_out(pl, n, units);
    if (pl.classes > kMaxClasses || pl.unit0[0] != 0 || pl.unit0[pl.classes] != units) return std::puts("classes"), 1;
    std::vector<double> load(units, 0.0);
    std::priority_queue<double, std::vector<double>, std::greater<double>> one_by_one;
    for (int u = 0; u < units; ++u) one_by_one.push(0.0);
    for (int k = 0; k < n; ++k) {
      std::vector<int> taken(pl.shape[k].tiles, 0);
      for (int c = 0; c < pl.classes; ++c) {
        const int width = pl.unit0[c + 1] - pl.unit0[c];
        for (int u = 0; u < width; ++u)
          for (int j = 0; j < pl.count[c][k]; ++j) {
            const int tile = pl.first[c][k] + j * width + u;         // as Walk::tile
            if (tile < 0 || tile >= (int)taken.size() || taken[tile]++) return std::puts("tile"), 1;
            if (pl.unit0[c] + u >= pl.units) return std::puts("unit"), 1;
            load[pl.unit0[c] + u] += pl.shape[k].cost;
          }
      }
      for (int t : taken)
        if (t != 1) return std::puts("left out"), 1;
      for (size_t t = 0; t < taken.size(); ++t) {
        const double least = one_by_one.top();
        one_by_one.pop();
        one_by_one.push(least + pl.shape[k].cost);
      }
    }
    double most = 0.0, best = 0.0;
    for (double l : load) most = std::max(most, l);
    for (; !one_by_one.empty(); one_by_one.pop()) best = one_by_one.top();
    if (std::abs(most - pl.makespan) > 1e-9 * best || most > best * (1.0 + 1e-9)) return std::printf("load %g %g\n", most, best), 1;
  }
  // the most rows of a launch: no unit's count leaves 16 bits
  for (int trial = 0; trial < 200; ++trial) {
    const int64_t columns = pick(0, 1) ? pick(1, 4096) : pick(1, 64), rows = zp_rows_per_launch(columns);
    GroupPlan pl;
    pl.shape[0].tiles = zp_ceil_div(rows, 128) * zp_ceil_div(columns, 64);
    pl.shape[0].cost = 4000;
    share_out(pl, 1, pick(64, 148));
    for (int c = 0; c < pl.classes; ++c)
      if (pl.count[c][0] > INT16_MAX) return std::puts("count"), 1;
  }
  std::puts("ok");
}
