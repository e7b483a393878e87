// Work items of the batched form: the regions of every enabled scene, in
// longest-processing-time order for the persistent raster grid.  Host code,
// shared by the renderer and its native tests.
#pragma once

#include <algorithm>
#include <cstdint>
#include <numeric>
#include <vector>

#include "records.h"

namespace gbr {

// What the ordering needs to know of a scene.
struct ItemScene {
  int width = 0, height = 0;  // viewport
  uint64_t tris = 0;          // drawn_tris() of the scene it renders (its source)
  uint32_t geometry = 0;      // groups items of equal cost (the mesh of the source's largest draw)
  bool enabled = true;
  uint32_t draws = 0;         // draws of that scene
  uint64_t all_tris = 0;      // all its triangles
};

// Region halvings a costly scene's items may get, and the most when the
// whole step has fewer items than the grid has CTAs.
constexpr int kMaxSplits = 4;
constexpr int kMaxFewSplits = 6;

// Region of a scene's items after `level` splits of the batched form's
// region (clamped to the viewport): each split halves the longer side, down
// to 32 pixels (16 beyond kMaxSplits).
inline void split_region(int width, int height, int region_w, int region_h, int level, int& rw, int& rh) {
  rw = std::max(1, std::min(region_w, width));
  rh = std::max(1, std::min(region_h, height));
  for (int l = 0; l < level; ++l) {
    const int side = l < kMaxSplits ? 32 : 16;
    if (rw >= rh && rw > side)
      rw = (rw + 1) / 2;
    else if (rh > side)
      rh = (rh + 1) / 2;
    else if (rw > side)
      rw = (rw + 1) / 2;
  }
}

// The same with upright strips: half the area a split, up to 128 rows, then 16
// columns and fewer rows.  The costly parts of a view lie side by side around its
// horizon, so that strips share them.  (The plain split where a strip would need
// more depth tiles than the whole region has.)
inline void split_region_tall(int width, int height, int region_w, int region_h, int level, int& rw, int& rh) {
  const int area = (region_w * region_h) >> level;
  rw = std::max(16, area / 128);
  rh = std::max(1, area / rw);
  const auto tiles = [](int w, int h, int side) { return ((w + side - 1) / side) * ((h + side - 1) / side); };
  if (area < 256 || tiles(rw, rh, 8) > tiles(region_w, region_h, 8) ||
      tiles(rw, rh, 32) > tiles(region_w, region_h, 32))
    return split_region(width, height, region_w, region_h, level, rw, rh);
  rw = std::max(1, std::min(rw, width));
  rh = std::max(1, std::min(rh, height));
}

// Triangles that a view of a scene draws, for item_cost: a camera sees most of
// a large draw around it, but few of many small draws.
inline uint64_t drawn_tris(uint64_t tris, uint64_t largest_draw) {
  return (26 * largest_draw + 7 * (tris - largest_draw)) / 20;
}

// Estimated cost of a w x h region of a W x H viewport in nanoseconds of a
// 512-thread CTA, two per SM: its share of the drawn triangles, 7 per pixel for
// rasterising and shading it, 18000 for the phases that every region goes
// through, a fiftieth of the triangles and 100 per draw for culling the scene.
// Fitted to the mean item of eight scene sets at five region sizes (bare and
// furnished rooms, scans, lit rooms; 128 x 64 to 16 x 32): within 10 % except
// lit rooms (half).
inline uint64_t item_cost(uint64_t tris, int w, int h, int W, int H, uint32_t draws = 0) {
  const uint64_t px = uint64_t(w) * uint64_t(h);
  return tris * px / (uint64_t(W) * uint64_t(H)) + 7 * px + 18000 + tris / 50 + 100 * uint64_t(draws);
}

// Estimated time of `items` items of total cost `total`, the largest costing
// `largest`, on `grid` CTAs, longest first: one wave ends with its longest item,
// several with a mean one.  The longest of equal estimates takes 2.5 times that
// (the views of a step differ that much).
inline double step_cost(uint64_t items, double total, double largest, uint64_t grid) {
  if (items <= grid) return 2.5 * largest;
  return std::max(2.5 * largest, total / double(grid) + 2.5 * total / double(items));
}

// Estimated cost of a w x h region where the longest item matters (lists that
// the device orders, the per-scene form): 0.9 for each triangle of its share of
// the scene, 11.5 per pixel, 30000, and 0.03 per triangle and 85 per draw for
// culling.  The triangles' part varies from view to view, and from region to
// region less where they span the view's height: `longest` adds as much of it
// as the longest of a step has.  (A factor on the whole cost, as in step_cost, is
// too small for furnished rooms or too large for bare ones.)
inline uint64_t region_cost(uint64_t tris, int w, int h, int W, int H, uint32_t draws, double& longest) {
  const uint64_t px = uint64_t(w) * uint64_t(h);
  const uint64_t part = 9 * tris * px / (10 * uint64_t(W) * uint64_t(H));
  const uint64_t cost = part + 23 * px / 2 + 30000 + 3 * tris / 100 + 85 * uint64_t(draws);
  longest = double(cost) + (h >= H ? 1.4 : 2.8) * double(part);
  return cost;
}

// Estimated time of such items on `grid` CTAs, the costliest first, of total cost
// `total`: one wave ends with its longest item, several when the work is done,
// with a little of it as the tail.  Strips (regions taller than 64 rows) take a
// twentieth more for what they draw twice.  With region_cost fitted to whole
// steps, 34 scene sets (bare and furnished rooms, scans, lit and mixed views; 4 to
// 1000 views) at nine sizes: the size with the least estimate is 1.2 % slower than
// the best on average (17 % at most).
inline double region_step_cost(uint64_t items, double total, double longest, uint64_t grid, bool strips) {
  const double time = items <= grid ? longest : std::max(longest, total / double(grid) + 0.1 * longest);
  return strips ? 1.05 * time : time;
}

// Items of one scene split `level` times and the cost of the largest.
inline void split_cost(const ItemScene& sc, int region_w, int region_h, int level, uint64_t& items, uint64_t& cost) {
  int rw, rh;
  split_region(sc.width, sc.height, region_w, region_h, level, rw, rh);
  items = uint64_t((sc.width + rw - 1) / rw) * uint64_t((sc.height + rh - 1) / rh);
  cost = item_cost(sc.tris, rw, rh, sc.width, sc.height, sc.draws);
}

// Items the list can ever hold: every scene at its finest split, plus the
// halves of the last wave (one per resident CTA, at most `max_grid`).
inline uint64_t work_item_capacity(const std::vector<ItemScene>& scenes, int region_w, int region_h,
                                   uint64_t max_grid) {
  uint64_t capacity = max_grid;
  for (const ItemScene& sc : scenes) {
    if (sc.width <= 0 || sc.height <= 0) continue;
    int rw, rh;
    split_region(sc.width, sc.height, region_w, region_h, kMaxSplits, rw, rh);
    capacity += uint64_t((sc.width + rw - 1) / rw) * uint64_t((sc.height + rh - 1) / rh);
  }
  return capacity;
}

// The items of the enabled scenes for a persistent grid of `grid` CTAs,
// longest first.  No item may cost more than a limit: a scene whose regions
// do gets them halved (at most kMaxSplits times, or kMaxFewSplits while the
// step has no more items than CTAs).  The limit, the largest whole region's
// cost or one of a falling sequence below it, is the one with the least
// step_cost: it breaks up a small viewport bound to a large scene beside light
// ones, and spreads a few views over the whole GPU.  Then the cheapest `grid` items --
// the last wave -- are halved (longer side, not below 32 px), so that the CTAs
// finishing the step wait for half an item at most.  Items of equal cost are
// grouped by geometry, so that the CTAs in flight read the same vertices from
// L2.  Halving two waves or quartering the last one was slower than halving
// one.
// order_capacity > 0: for a list that the device orders (its keys see the
// cameras), if that many items hold it: the limit by region_cost, regions or
// upright strips by the same estimate, no halving of the last wave (it only adds
// items: 1024 textured views 1617 -> 1653 us with it), the items in scene order,
// each scene's regions row by row.
inline std::vector<WorkItem> build_work_items(const std::vector<ItemScene>& scenes, int region_w, int region_h,
                                              uint64_t grid, uint64_t order_capacity = 0) {
  const bool ordered = order_capacity > 0;
  grid = std::max<uint64_t>(grid, 1);
  std::vector<uint32_t> on;  // the scenes that have items
  for (uint32_t s = 0; s < scenes.size(); ++s)
    if (scenes[s].enabled && scenes[s].width > 0 && scenes[s].height > 0) on.push_back(s);
  // Per such scene and level, whole regions and strips: items and largest cost
  // (levels that change nothing repeat).
  struct Level {
    uint64_t items, cost;
    double longest;
  };
  const int deepest = ordered ? kMaxSplits : kMaxFewSplits;
  std::vector<Level> levels[2];
  auto level_of = [&](size_t n, bool strips, uint64_t t, int most) {
    const Level* l = &levels[strips][n * size_t(deepest + 1)];
    int k = 0;
    while (k < most && l[k].cost > t) ++k;
    return k;
  };
  int max_splits = kMaxSplits;
  double best = -1.0;
  uint64_t best_limit = 0;
  bool tall = false;
  auto region = [&](uint32_t s, int level, bool strips, int& rw, int& rh) {
    // (Whole regions stay as they are; 32 x 32 regions are worse than strips.)
    ((strips && level > 0) || (ordered && level > 2) ? split_region_tall : split_region)(
        scenes[s].width, scenes[s].height, region_w, region_h, level, rw, rh);
  };
  for (const bool strips : {false, true}) {
    if (strips && !ordered) break;
    uint64_t limit = 1;
    levels[strips].resize(on.size() * size_t(deepest + 1), Level{0, 0, 0.0});
    for (size_t n = 0; n < on.size(); ++n) {
      const ItemScene& sc = scenes[on[n]];
      Level* l = &levels[strips][n * size_t(deepest + 1)];
      for (int k = 0; k <= deepest; ++k) {
        if (!ordered) {
          split_cost(sc, region_w, region_h, k, l[k].items, l[k].cost);
          continue;
        }
        int rw, rh;
        region(on[n], k, strips, rw, rh);
        l[k].items = uint64_t((sc.width + rw - 1) / rw) * uint64_t((sc.height + rh - 1) / rh);
        l[k].cost = region_cost(std::max(sc.all_tris, sc.tris), rw, rh, sc.width, sc.height, sc.draws, l[k].longest);
      }
      limit = std::max(limit, l[0].cost);
    }
    for (int most : {kMaxSplits, kMaxFewSplits}) {
      if (ordered && most > kMaxSplits) break;
      uint64_t t = limit;
      for (int i = 0; i < 28 && t > 0; ++i, t = t * 17 / 20) {
        uint64_t items = 0, total = 0, largest = 0;
        double longest = 0.0;
        bool few = false;
        for (size_t n = 0; n < on.size(); ++n) {
          const Level* l = &levels[strips][n * size_t(deepest + 1)];
          const int k = level_of(n, strips, t, most);
          few = few || k > kMaxSplits;
          items += l[k].items;
          total += l[k].items * l[k].cost;
          largest = std::max(largest, l[k].cost);
          longest = std::max(longest, l[k].longest);
        }
        if (few && items > grid) break;
        if (ordered && i > 0 && items > order_capacity) break;
        const double cost = ordered ? region_step_cost(items, double(total), longest, grid, strips)
                                    : step_cost(items, double(total), double(largest), grid);
        if (best < 0.0 || cost < best) {
          best = cost;
          best_limit = t;
          max_splits = most;
          tall = strips;
        }
      }
    }
  }
  std::vector<WorkItem> items;
  std::vector<uint64_t> cost;
  std::vector<uint32_t> key;
  for (size_t n = 0; n < on.size(); ++n) {
    const uint32_t s = on[n];
    const ItemScene& sc = scenes[s];
    int rw, rh;
    region(s, level_of(n, tall, best_limit, max_splits), tall, rw, rh);
    for (int y = 0; y < sc.height; y += rh)
      for (int x = 0; x < sc.width; x += rw) {
        WorkItem it{};
        it.scene = s;
        it.x0 = uint16_t(x);
        it.y0 = uint16_t(y);
        it.w = uint16_t(std::min(rw, sc.width - x));
        it.h = uint16_t(std::min(rh, sc.height - y));
        items.push_back(it);
        cost.push_back(item_cost(sc.tris, it.w, it.h, sc.width, sc.height, sc.draws));
        key.push_back(sc.geometry);
      }
  }
  if (ordered) return items;
  std::vector<uint32_t> perm(items.size());
  std::iota(perm.begin(), perm.end(), 0u);
  auto by_cost = [&](uint32_t a, uint32_t b) {
    if (cost[a] != cost[b]) return cost[a] > cost[b];
    return key[a] < key[b];
  };
  std::stable_sort(perm.begin(), perm.end(), by_cost);
  if (items.size() > grid) {
    const size_t n0 = items.size();
    for (size_t i = n0 - grid; i < n0; ++i) {
      WorkItem& it = items[perm[i]];
      WorkItem b = it;
      if (it.w >= it.h && it.w > 32) {
        b.w = uint16_t(it.w / 2);
        b.x0 = uint16_t(it.x0 + (it.w - b.w));
        it.w = uint16_t(it.w - b.w);
      } else if (it.h > 32) {
        b.h = uint16_t(it.h / 2);
        b.y0 = uint16_t(it.y0 + (it.h - b.h));
        it.h = uint16_t(it.h - b.h);
      } else {
        continue;
      }
      const ItemScene& sc = scenes[it.scene];
      const uint32_t geometry = key[perm[i]];
      cost[perm[i]] = item_cost(sc.tris, it.w, it.h, sc.width, sc.height, sc.draws);
      const uint64_t bcost = item_cost(sc.tris, b.w, b.h, sc.width, sc.height, sc.draws);
      items.push_back(b);  // `it` is not used past this point
      cost.push_back(bcost);
      key.push_back(geometry);
    }
    perm.resize(items.size());
    std::iota(perm.begin(), perm.end(), 0u);
    std::stable_sort(perm.begin(), perm.end(), by_cost);
  }
  std::vector<WorkItem> out(items.size());
  for (size_t i = 0; i < items.size(); ++i) out[i] = items[perm[i]];
  return out;
}

}  // namespace gbr
