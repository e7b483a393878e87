// The plan of a step (work_items.h): scenes of one size and cost are one class and
// are cut alike, whatever their order; the plan counts the items that its list
// holds (before the last wave is halved), so that a list is made once.
#include <cuda_runtime.h>

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

int main() {
  std::mt19937_64 rng(11);
  for (int trial = 0; trial < 200; ++trial) {
    std::vector<ItemScene> kinds(1 + rng() % 8);
    for (ItemScene& k : kinds) {
      k.width = 1 + int(rng() % 300);
      k.height = 1 + int(rng() % 300);
      k.tris = rng() % 400000;
      k.all_tris = k.tris + rng() % 1000;
      k.draws = uint32_t(rng() % 200);
    }
    std::vector<ItemScene> scenes(rng() % 600);
    std::vector<uint32_t> kind(scenes.size());
    for (size_t s = 0; s < scenes.size(); ++s) {
      scenes[s] = kinds[kind[s] = uint32_t(rng() % kinds.size())];
      scenes[s].geometry = uint32_t(rng() % 9);
      scenes[s].enabled = rng() % 4 != 0;
    }
    for (const bool ordered : {false, true}) {
      const uint64_t capacity = ordered ? 1 + work_item_capacity(scenes, 128, 64, 304) * 3 / 7 : 0;
      const ItemPlan plan = plan_work_items(scenes, 128, 64, 304, capacity);
      CHECK(plan.classes.size() <= kinds.size());
      uint64_t items = 0, of_classes = 0;
      for (const ItemClass& c : plan.classes) {
        CHECK(c.rw >= 1 && c.rh >= 1 && c.rw * c.rh <= 128 * 64);
        items += uint64_t((c.width + c.rw - 1) / c.rw) * uint64_t((c.height + c.rh - 1) / c.rh) * c.scenes;
        of_classes += c.scenes;
      }
      CHECK(items == plan.items && of_classes == plan.on.size());
      for (size_t n = 0; n < plan.on.size(); ++n) {
        const ItemScene& sc = scenes[plan.on[n]];
        const ItemClass& c = plan.classes[plan.class_of[n]];
        CHECK(sc.enabled && c.width == sc.width && c.height == sc.height && c.tris == sc.tris);
      }
      const size_t list = emit_work_items(plan, scenes, 304).size();
      CHECK(ordered || items > 304 ? list >= items && list <= items + 304 : list == items);
      CHECK(!ordered || list == items);
    }
  }
  if (failures) return 1;
  std::printf("ok\n");
  return 0;
}
