// Sharing the tiles of a launch's products out among the CTAs (zp_gemm_tc.cu).  Host code.
#pragma once

#include <algorithm>
#include <cmath>
#include <cstdint>

#include "zp_common.cuh"

// Units (CTAs, or CTA pairs) that take the same number of tiles of each product; one more class than products
constexpr int kMaxClasses = ZP_GEMM_GROUP + 1;

// How the products of one launch are cut into tiles and shared out.
struct Shape {
  int bn, num_n, ksplit, kbs, num_k;
  int64_t tiles;
  double cost;                           // of one tile, in SM clocks or so
};
struct GroupPlan {
  int order[ZP_GEMM_GROUP];              // products, longest tiles first
  Shape shape[ZP_GEMM_GROUP];            // in that order
  int classes, unit0[kMaxClasses + 1], first[kMaxClasses][ZP_GEMM_GROUP], count[kMaxClasses][ZP_GEMM_GROUP];
  bool pair;
  int bk, halves;                        // depth of a k-block; CTAs that share a B tile
  int max_bn, units;                     // units that have work
  double makespan;
};

// A unit's tiles of a product are counted in 16 bits (a launch's parameters in 32 cost every small launch 0.2 us):
// so many rows of tiles of at least 64 columns, on 64 units or more, one launch takes.
inline int64_t zp_rows_per_launch(int64_t columns) {
  return std::max<int64_t>(INT16_MAX / zp_ceil_div(columns, 64), 1) * 64 * 128;
}

// Shares the tiles out: products in turn, longest tiles first, every tile to a unit that has least so far.
// Units that stand alike are a class and treated as one, so this takes a microsecond and not one per tile.
// A fixed stride through the list gave the same units the longest tiles of every round.  With this, and the
// kernels' set-up beside the kernel before them: 200 atoms in bf16 294 -> 280 us (inference), 500 in two planes
// 2 900 -> 2 770 and 777 of ragged widths in three 1 316 -> 1 269 (training steps).
inline void share_out(GroupPlan &pl, int n, int units) {
  double load[kMaxClasses] = {0.0};
  int classes = 1;
  pl.unit0[0] = 0;
  pl.unit0[1] = units;
  for (int k = 0; k < n; ++k) {
    for (int c = 0; c < classes; ++c) pl.count[c][k] = 0;
    int64_t left = pl.shape[k].tiles;
    const double cost = pl.shape[k].cost;
    while (left > 0) {
      int low = 0;
      for (int c = 1; c < classes; ++c)
        if (load[c] < load[low]) low = c;
      double next = 1e300;               // load of the next class up
      for (int c = 0; c < classes; ++c)
        if (c != low && load[c] < next) next = load[c];
      const int64_t width = pl.unit0[low + 1] - pl.unit0[low];
      if (left >= width) {
        int64_t rounds = left / width;
        if (next < 1e300) rounds = std::min(rounds, std::max<int64_t>(1, (int64_t)std::ceil((next - load[low]) / cost)));
        pl.count[low][k] += (int)rounds;
        load[low] += (double)rounds * cost;
        left -= rounds * width;
        continue;
      }
      for (int c = classes; c > low; --c) {      // the first `left` units of the class take one more
        pl.unit0[c + 1] = pl.unit0[c];
        load[c] = load[c - 1];
        for (int i = 0; i <= k; ++i) pl.count[c][i] = pl.count[c - 1][i];
      }
      ++classes;
      pl.unit0[low + 1] = pl.unit0[low] + (int)left;
      pl.count[low][k] += 1;
      load[low] += cost;
      left = 0;
    }
  }
  pl.classes = classes;
  pl.units = 0;
  pl.makespan = 0.0;
  for (int c = 0; c < classes; ++c) {
    if (load[c] > 0.0) pl.units = pl.unit0[c + 1];
    pl.makespan = std::max(pl.makespan, load[c]);
  }
  for (int k = 0; k < n; ++k) {
    int at = 0;
    for (int c = 0; c < classes; ++c) {
      pl.first[c][k] = at;
      at += pl.count[c][k] * (pl.unit0[c + 1] - pl.unit0[c]);
    }
  }
}
