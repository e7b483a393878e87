// The per-scene form over some of a renderer's scenes: its list holds the drawn
// scenes' regions and no others, in regions chosen for those scenes, whatever
// else the renderer holds; a caller's regions are kept.
#include "renderer.cpp"

#include <random>

#include "fake_cuda.h"

using namespace gbr;

struct Launch {
  uint32_t grid = 0;
  int w = 0, h = 0;
};

static Launch last;
static std::vector<uint8_t> drawn;
static int width, height;

static void watch() {
  fake::on_raster = [](const RasterParams& p, int, uint32_t grid, size_t smem) {
    if (p.persistent) return;  // a batched draw between
    last = {grid, p.region_w, p.region_h};
    CHECK(p.item_count == grid);
    if (p.item_base) return;  // ordered: the sorted list is the kernel's
    std::vector<uint64_t> px(drawn.size());
    for (uint32_t i = 0; i < grid; ++i) {
      const WorkItem& it = p.items[i];
      CHECK(it.scene < drawn.size() && drawn[it.scene]);
      CHECK(p.cameras[it.scene].enabled >= 1 && p.cameras[it.scene].enabled - 1 <= i);
      CHECK(it.w <= p.region_w && it.h <= p.region_h);
      px[it.scene] += uint64_t(it.w) * it.h;
    }
    for (size_t s = 0; s < px.size(); ++s)
      CHECK(px[s] == (drawn[s] ? uint64_t(width) * uint64_t(height) : 0));
  };
}

static Launch draw(Renderer* r, cudaStream_t stream, uint32_t on) {
  for (uint32_t s = 0; s < drawn.size(); ++s) {
    drawn[s] = s * 7 % drawn.size() < on;
    CHECK(r->set_enabled(s, drawn[s]) == GBR_OK);
  }
  last = {};
  CHECK(r->draw(stream, GBR_DRAW_PER_SCENE, false) == GBR_OK);
  return last;
}

int main() {
  width = height = 128;
  const cudaStream_t stream = fake::stream(false);
  drawn.assign(1, 1);
  Renderer* one = fake::renderer(1, width, height, 50);
  watch();
  const Launch alone = draw(one, stream, 1);
  delete one;

  drawn.assign(1024, 1);
  Renderer* many = fake::renderer(1024, width, height, 50);
  const Launch all = draw(many, stream, 1024);
  CHECK(all.grid >= 1024);
  const Launch few = draw(many, stream, 1);
  CHECK(few.grid == alone.grid && few.w == alone.w && few.h == alone.h);
  CHECK(draw(many, stream, 0).grid == 0);
  std::mt19937 rng(5);
  for (int k = 0; k < 30; ++k) {
    draw(many, stream, rng() % 1025);
    if (k % 4 == 0) CHECK(many->draw(stream, GBR_DRAW_BATCHED, true) == GBR_OK);
    fake::run_legacy();
  }
  gbr_tuning t{1024, 128, 128, 1, 1, 24, 40, 1, 75};
  CHECK(many->set_tuning(t) == GBR_OK);
  const Launch tuned = draw(many, stream, 3);
  CHECK(tuned.w == 24 && tuned.h == 40 && tuned.grid == 3 * 6 * 4);
  delete many;
  return fake::finish();
}
