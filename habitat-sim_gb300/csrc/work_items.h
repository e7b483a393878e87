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

// Scenes that are cut alike: of one size and cost.
struct ItemClass {
  int width, height;
  uint64_t tris, all_tris;
  uint32_t draws;
  uint32_t scenes;  // how many
  int rw, rh;       // the region chosen for them
};

// How a step is cut.
struct ItemPlan {
  std::vector<uint32_t> on;        // the scenes that have items
  std::vector<uint32_t> class_of;  // of each of those
  std::vector<ItemClass> classes;
  uint64_t items = 0;
  bool ordered = false;
};

// The regions of the enabled scenes for a persistent grid of `grid` CTAs.  No
// item may cost more than a limit: a scene whose regions do gets them halved (at
// most kMaxSplits times, or kMaxFewSplits while the step has no more items than
// CTAs).  The limit, the largest whole region's cost or one of a falling sequence
// below it, is the one with the least step_cost: it breaks up a small viewport
// bound to a large scene beside light ones, and spreads a few views over the
// whole GPU.
// order_capacity > 0: for a list that the device orders (its keys see the
// cameras), if that many items hold it: the limit by region_cost, regions or
// upright strips by the same estimate.
//
// Made again whenever the drawn scenes change, on the path of a server's step,
// so it goes by classes of scenes, and down the limits each class moves from
// level to level once: with the list, 1024 views of 4 scenes take 50 us and of
// 24 at three sizes 65 (an x86 core); scene by scene, 235 and 551.
inline ItemPlan plan_work_items(const std::vector<ItemScene>& scenes, int region_w, int region_h, uint64_t grid,
                                uint64_t order_capacity = 0) {
  ItemPlan plan;
  const bool ordered = plan.ordered = order_capacity > 0;
  grid = std::max<uint64_t>(grid, 1);
  std::vector<ItemClass>& classes = plan.classes;
  size_t slots = 16;
  while (slots < 2 * scenes.size()) slots *= 2;
  std::vector<uint32_t> table(slots, 0xffffffffu);
  plan.on.reserve(scenes.size());
  plan.class_of.reserve(scenes.size());
  for (uint32_t s = 0; s < scenes.size(); ++s) {
    const ItemScene& sc = scenes[s];
    if (!sc.enabled || sc.width <= 0 || sc.height <= 0) continue;
    uint64_t h = sc.tris;
    for (const uint64_t v : {uint64_t(sc.all_tris), uint64_t(sc.draws), uint64_t(sc.width) << 32 | uint32_t(sc.height)})
      h = (h ^ (h >> 29)) * 0x9e3779b97f4a7c15ull + v;
    h = (h ^ (h >> 32)) * 0x9e3779b97f4a7c15ull;
    size_t at = size_t(h >> 20) & (slots - 1);
    for (;; at = (at + 1) & (slots - 1)) {
      if (table[at] == 0xffffffffu) {
        table[at] = uint32_t(classes.size());
        classes.push_back({sc.width, sc.height, sc.tris, sc.all_tris, sc.draws, 0, 0, 0});
        break;
      }
      const ItemClass& c = classes[table[at]];
      if (c.width == sc.width && c.height == sc.height && c.tris == sc.tris && c.all_tris == sc.all_tris &&
          c.draws == sc.draws)
        break;
    }
    ++classes[table[at]].scenes;
    plan.on.push_back(s);
    plan.class_of.push_back(table[at]);
  }
  // Per class and level, whole regions and strips: items of all its scenes and
  // largest cost (levels that change nothing repeat).
  struct Level {
    uint64_t items, cost;
    double longest;
  };
  const size_t C = classes.size();
  const int deepest = ordered ? kMaxSplits : kMaxFewSplits;
  std::vector<Level> levels[2];
  int max_splits = kMaxSplits;
  double best = -1.0;
  uint64_t best_limit = 0;
  bool tall = false;
  auto region = [&](const ItemClass& c, int level, bool strips, int& rw, int& rh) {
    // (Whole regions stay as they are; 32 x 32 regions are worse than strips.)
    ((strips && level > 0) || (ordered && level > 2) ? split_region_tall : split_region)(c.width, c.height, region_w,
                                                                                         region_h, level, rw, rh);
  };
  std::vector<uint8_t> at(C);            // level of each class at the limit
  std::vector<uint64_t> cost_at(C);      // and what it costs there
  std::vector<double> longest_at(C);
  for (const bool strips : {false, true}) {
    if (strips && !ordered) break;
    uint64_t limit = 1;
    levels[strips].resize(C * size_t(deepest + 1), Level{0, 0, 0.0});
    for (size_t n = 0; n < C; ++n) {
      const ItemClass& c = classes[n];
      Level* l = &levels[strips][n * size_t(deepest + 1)];
      for (int k = 0; k <= deepest; ++k) {
        int rw, rh;
        region(c, k, strips, rw, rh);
        l[k].items = uint64_t((c.width + rw - 1) / rw) * uint64_t((c.height + rh - 1) / rh) * c.scenes;
        l[k].cost = ordered ? region_cost(std::max(c.all_tris, c.tris), rw, rh, c.width, c.height, c.draws, l[k].longest)
                            : item_cost(c.tris, rw, rh, c.width, c.height, c.draws);
      }
      limit = std::max(limit, l[0].cost);
    }
    for (int most : {kMaxSplits, kMaxFewSplits}) {
      if (ordered && most > kMaxSplits) break;
      uint64_t items = 0, total = 0;
      bool few = false;
      for (size_t n = 0; n < C; ++n) {
        const Level& l = levels[strips][n * size_t(deepest + 1)];
        at[n] = 0;
        cost_at[n] = l.cost;
        longest_at[n] = l.longest;
        items += l.items;
        total += l.items * l.cost;
      }
      uint64_t t = limit;
      for (int i = 0; i < 28 && t > 0; ++i, t = t * 17 / 20) {
        uint64_t largest = 0;
        double longest = 0.0;
        for (size_t n = 0; n < C; ++n) {
          if (cost_at[n] > t && at[n] < most) {
            const Level* l = &levels[strips][n * size_t(deepest + 1)];
            int k = at[n];
            items -= l[k].items;
            total -= l[k].items * l[k].cost;
            while (k < most && l[k].cost > t) ++k;
            items += l[k].items;
            total += l[k].items * l[k].cost;
            few = few || k > kMaxSplits;
            at[n] = uint8_t(k);
            cost_at[n] = l[k].cost;
            longest_at[n] = l[k].longest;
          }
          largest = std::max(largest, cost_at[n]);
          longest = std::max(longest, longest_at[n]);
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
          plan.items = items;
        }
      }
    }
  }
  for (size_t n = 0; n < C; ++n) {
    const Level* l = &levels[tall][n * size_t(deepest + 1)];
    int k = 0;
    while (k < max_splits && l[k].cost > best_limit) ++k;
    region(classes[n], k, tall, classes[n].rw, classes[n].rh);
  }
  return plan;
}

// The plan's items.  For a list that the device orders: in scene order, each
// scene's regions row by row.  Else longest first, and the cheapest `grid` items
// -- the last wave -- halved (longer side, not below 32 px), so that the CTAs
// finishing the step wait for half an item at most.  Items of equal cost are
// grouped by geometry, so that the CTAs in flight read the same vertices from
// L2.  Halving two waves or quartering the last one was slower than halving one;
// in an ordered list it only adds items (1024 textured views 1617 -> 1653 us).
inline std::vector<WorkItem> emit_work_items(const ItemPlan& plan, const std::vector<ItemScene>& scenes, uint64_t grid) {
  grid = std::max<uint64_t>(grid, 1);
  std::vector<WorkItem> items;
  std::vector<uint64_t> cost;
  std::vector<uint32_t> key;
  items.reserve(plan.items + (plan.ordered ? 0 : grid));
  if (!plan.ordered) {
    cost.reserve(plan.items + grid);
    key.reserve(plan.items + grid);
  }
  for (size_t n = 0; n < plan.on.size(); ++n) {
    const uint32_t s = plan.on[n];
    const ItemScene& sc = scenes[s];
    const int rw = plan.classes[plan.class_of[n]].rw, rh = plan.classes[plan.class_of[n]].rh;
    for (int y = 0; y < sc.height; y += rh)
      for (int x = 0; x < sc.width; x += rw) {
        WorkItem it{};
        it.scene = s;
        it.x0 = uint16_t(x);
        it.y0 = uint16_t(y);
        it.w = uint16_t(std::min(rw, sc.width - x));
        it.h = uint16_t(std::min(rh, sc.height - y));
        items.push_back(it);
        if (plan.ordered) continue;
        cost.push_back(item_cost(sc.tris, it.w, it.h, sc.width, sc.height, sc.draws));
        key.push_back(sc.geometry);
      }
  }
  if (plan.ordered) return items;
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

inline std::vector<WorkItem> build_work_items(const std::vector<ItemScene>& scenes, int region_w, int region_h,
                                              uint64_t grid, uint64_t order_capacity = 0) {
  return emit_work_items(plan_work_items(scenes, region_w, region_h, grid, order_capacity), scenes, grid);
}

}  // namespace gbr
