// Lists for the device to order (work_items.h): on random scene sets, every
// enabled viewport covered exactly once, a scene's items contiguous and row by
// row, all but the last of a row or column of the first one's size, split
// only as far as the list has room.
#include <cuda_runtime.h>

#include <cmath>
#include <cstdio>
#include <random>
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

static void check_set(const std::vector<ItemScene>& scenes, int rw, int rh, uint64_t grid) {
  const uint64_t room = work_item_capacity(scenes, rw, rh, grid), part = room * 3 / 7;
  const std::vector<WorkItem> items = build_work_items(scenes, rw, rh, grid, part);
  CHECK(items.size() <= room);
  uint64_t whole = 0;
  for (const ItemScene& sc : scenes)
    if (sc.enabled) whole += uint64_t((sc.width + rw - 1) / rw) * uint64_t((sc.height + rh - 1) / rh);
  CHECK(items.size() <= std::max(part, whole));  // split only as far as there is room
  size_t i = 0;
  for (uint32_t s = 0; s < scenes.size(); ++s) {
    if (!scenes[s].enabled) continue;
    CHECK(i < items.size() && items[i].scene == s);
    if (i >= items.size()) return;
    const int W = scenes[s].width, H = scenes[s].height, w = items[i].w, h = items[i].h;
    CHECK(w >= 1 && h >= 1 && w * h <= rw * rh);
    const auto tiles = [](int x, int y, int side) { return ((x + side - 1) / side) * ((y + side - 1) / side); };
    CHECK(tiles(w, h, 8) <= tiles(rw, rh, 8) && tiles(w, h, 32) <= tiles(rw, rh, 32));  // room for the depth tiles
    for (int y = 0; y < H; y += h)
      for (int x = 0; x < W; x += w, ++i) {
        CHECK(i < items.size());
        if (i >= items.size()) return;
        const WorkItem& it = items[i];
        CHECK(it.scene == s && it.x0 == x && it.y0 == y);
        CHECK(it.w == std::min(w, W - x) && it.h == std::min(h, H - y));
      }
  }
  CHECK(i == items.size());
}

int main() {
  std::mt19937_64 rng(43);
  const int shapes[][2] = {{128, 128}, {128, 64}, {64, 64}, {32, 32}};
  const uint64_t grids[] = {1, 152, 304, 608};
  for (int trial = 0; trial < 300; ++trial) {
    std::vector<ItemScene> scenes(1 + rng() % 200);
    for (ItemScene& sc : scenes) {
      sc.width = 1 + int(rng() % 300);
      sc.height = 1 + int(rng() % 300);
      sc.tris = uint64_t(std::exp(std::uniform_real_distribution<double>(0.0, 15.0)(rng)));
      sc.draws = uint32_t(rng() % 300);
      sc.enabled = rng() % 5 != 0;
    }
    check_set(scenes, shapes[trial % 4][0], shapes[trial % 4][1], grids[trial / 4 % 4]);
  }
  CHECK(build_work_items({}, 128, 64, 304, 1).empty());
  if (failures) return 1;
  std::printf("ok\n");
  return 0;
}
