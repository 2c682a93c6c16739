// Work plans of the persistent tile kernels (forward and the adjoint's
// backward).
#pragma once

#include <algorithm>
#include <cmath>
#include <vector>

#include "bimp_internal.h"

namespace bimp_b200 {

// Cost of a work item: `item` for what it does once, and per orientation
// `orientation` + `block` for each block of four rows (of the rows inside the
// map) on the scheduler with most of them.
struct TileCost {
  double item, orientation, block;
};
// Fits to measured times, in units of one orientation of a V = 100 tile.
// Forward (1080p, residual 1.7 k of about 90 k cycles an item): 14.5 k, 5.0 k,
// 0.77 k of 10.4 k cycles.  The weights before the x-passes went warp by warp
// left a 3840 x 2160 detection's tile kernel at 946 us, these 859.
constexpr TileCost kForwardCost = {1.4, 0.481, 0.0741};
// Forward with the pipelined kernel, whose row and column passes overlap: of
// eleven sets of weights over eight batches of 3 to 24 images, the one with the
// shortest times (geometric mean 169.3 us; 175.5 with the weights above, up to
// 13% apart in a batch).
constexpr TileCost kPipelinedCost = {1.35, 0.70, 0.04};
// Backward (16 x 512 x 512, residual 11 k of about 300 k cycles an item): 61 k,
// 19.2 k, 1.68 k of 31.0 k cycles.
constexpr TileCost kBackwardCost = {1.97, 0.62, 0.0543};
// Backward from kept responses (between that case, 40.8 k, 13.4 k, 1.30 k, and
// 1333 x 1001, 35.9 k, 15.3 k, 1.08 k of 22.5 k cycles; residual 10 k of about
// 210 k).  The y-passes through tensor memory made an orientation 1.4 k cycles
// shorter; weights refitted to that moved the two cases' backward by +1.2% and
// -0.4%, so these stayed.
constexpr TileCost kBackwardKeptCost = {1.75, 0.62, 0.0535};

// Balanced plan for a persistent grid of `grid` CTAs.  The (tile,
// orientation) pairs, tile by tile in the given order, are cut into at most
// `grid` contiguous runs of about equal cost; a run becomes one work item
// per tile it touches (a tile cut between two CTAs is transformed forward by
// both).  The smallest run bound that fits in `grid` runs is found by
// bisection.  Item k of CTA b is placed at index k * grid + b (the kernels
// stride their work list by the grid); CTAs with fewer items get empty ones.
// *usedGrid receives the number of CTAs with work.
inline std::vector<TileWork> split_plan(const std::vector<TileWork>& tiles, const std::vector<ScaleDev>& sds,
                                        const TileCost& cost, int grid, int* usedGrid) {
  std::vector<double> ori(tiles.size());
  double total = 0.0, worst = 0.0;
  for (size_t i = 0; i < tiles.size(); ++i) {
    const ScaleDev& d = sds[tiles[i].entry];
    const int ty = tiles[i].tile / d.tilesX;
    const int vr = std::min(d.V, d.cRows - ty * d.V);   // valid rows inside the map (the x-passes' rows)
    const int blocks = ((vr + 3) / 4 + 3) / 4;   // four-row blocks of the busiest scheduler
    ori[i] = cost.orientation + cost.block * blocks;
    total += kNumOri * ori[i] + cost.item;
    worst = std::max(worst, ori[i] + cost.item);
  }
  // greedy runs of the pair sequence under bound tau (a pair joins the
  // current run while the run stays within tau); returns the run count
  auto cut = [&](double tau, std::vector<std::vector<TileWork>>* runs) {
    int n = 0;
    double acc = 0.0;
    for (size_t i = 0; i < tiles.size(); ++i)
      for (int o = 0; o < kNumOri;) {
        if (n == 0 || (acc + cost.item + ori[i] > tau && acc > 0.0)) {
          ++n;
          acc = 0.0;
          if (runs) runs->emplace_back();
        }
        acc += cost.item + ori[i];   // the item's forward transform and first orientation
        int k = 1 + static_cast<int>(std::floor(std::max(0.0, tau - acc) / ori[i]));
        k = std::min(k, kNumOri - o);
        acc += (k - 1) * ori[i];
        if (runs) runs->back().push_back({tiles[i].entry, tiles[i].tile, o, o + k});
        o += k;
      }
    return n;
  };
  double lo = std::max(worst, total / std::max(1, grid)) * 0.999, hi = total + worst;
  for (int it = 0; it < 60 && hi - lo > 1e-6 * hi; ++it) {
    const double mid = 0.5 * (lo + hi);
    if (cut(mid, nullptr) <= grid) hi = mid;
    else lo = mid;
  }
  std::vector<std::vector<TileWork>> runs;
  cut(hi, &runs);
  const int g = static_cast<int>(runs.size());
  size_t depth = 0;
  for (auto& r : runs) depth = std::max(depth, r.size());
  std::vector<TileWork> out(depth * (size_t)g, TileWork{0, 0, 0, 0});
  for (int b = 0; b < g; ++b)
    for (size_t k = 0; k < runs[b].size(); ++k) out[k * (size_t)g + b] = runs[b][k];
  *usedGrid = g;
  return out;
}

}  // namespace bimp_b200
