// Work items of steps with few views (work_items.h): every viewport covered
// exactly once within the list's capacity, as many items as keep the GPU busy
// but no more than its CTAs when the regions are split beyond kMaxSplits, and
// no further splitting once the step fills the grid.
#include <cuda_runtime.h>

#include <cstdio>
#include <vector>

#include "work_items.h"

using namespace gbr;

static int failures = 0;
#define CHECK(c)                                                   \
  do {                                                             \
    if (!(c)) {                                                    \
      std::fprintf(stderr, "%s:%d: %s\n", __FILE__, __LINE__, #c); \
      ++failures;                                                  \
    }                                                              \
  } while (0)

static std::vector<WorkItem> covered(const std::vector<ItemScene>& scenes, uint64_t grid) {
  const std::vector<WorkItem> items = build_work_items(scenes, 128, 64, grid);
  CHECK(items.size() <= work_item_capacity(scenes, 128, 64, grid));
  std::vector<std::vector<int>> hits(scenes.size());
  for (size_t s = 0; s < scenes.size(); ++s) hits[s].assign(size_t(scenes[s].width) * scenes[s].height, 0);
  for (const WorkItem& it : items)
    for (int y = it.y0; y < it.y0 + it.h; ++y)
      for (int x = it.x0; x < it.x0 + it.w; ++x) ++hits[it.scene][size_t(y) * scenes[it.scene].width + x];
  for (const auto& h : hits)
    for (int n : h) CHECK(n == 1);
  return items;
}

int main() {
  const uint64_t grids[] = {152, 304};
  for (uint64_t grid : grids) {
    for (int side : {1, 15, 16, 17, 33, 100, 128, 300}) {
      for (int n : {1, 2, 3, 16, 40}) {
        const auto items = covered(std::vector<ItemScene>(size_t(n), ItemScene{side, side, 50000, 0, true}), grid);
        int w = 0, h = 0;
        for (const WorkItem& it : items) {
          w = std::max<int>(w, it.w);
          h = std::max<int>(h, it.h);
        }
        if (w < 32 && h < 32 && side >= 64) CHECK(items.size() <= grid);  // beyond kMaxSplits
      }
    }
    // One 128 x 128 view spreads over at least 16 CTAs, 16 views over more
    // than half of the grid; 1000 views keep whole regions (and the halves
    // of the last wave).
    CHECK(covered({ItemScene{128, 128, 50000, 0, true}}, grid).size() >= 16);
    CHECK(covered(std::vector<ItemScene>(16, ItemScene{128, 128, 50000, 0, true}), grid).size() >= grid / 2);
    CHECK(covered(std::vector<ItemScene>(1000, ItemScene{128, 128, 50000, 0, true}), grid).size() == 2000 + grid);
  }
  // Nothing to draw, scenes without triangles, disabled scenes.
  CHECK(build_work_items({}, 128, 64, 304).empty());
  covered({ItemScene{64, 64, 0, 0, true}, ItemScene{1, 1, 0, 0, true}}, 304);
  CHECK(build_work_items({ItemScene{64, 64, 10, 0, false}}, 128, 64, 304).empty());
  // The shift of packed triangle ordinals: draw and triangle index in 32 bits.
  CHECK(ordinal_shift(1, 0) == 0 && ordinal_shift(1, 1) == 0 && ordinal_shift(200, 5000) == 13);
  CHECK(ordinal_shift(1, 1u << 31) == 31 && ordinal_shift(2, 1u << 31) == 31);
  CHECK(ordinal_shift(3, 1u << 31) == kOrdinalRunning && ordinal_shift(2, (1u << 31) + 1) == kOrdinalRunning);
  CHECK(ordinal_shift(2048, 1u << 21) == 21 && ordinal_shift(2049, 1u << 21) == kOrdinalRunning);
  if (failures) return 1;
  std::printf("ok\n");
  return 0;
}
