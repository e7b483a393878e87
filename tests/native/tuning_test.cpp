// Tuning by field: a field that the caller sets stays, the others are the
// library's choice whenever the caller asks or sets another one, and what is
// reported before the first draw is what the draw uses.
#include "renderer.cpp"

#include "fake_cuda.h"

using namespace gbr;

static gbr_tuning get(Renderer* r) {
  gbr_tuning t;
  CHECK(r->get_tuning(&t) == GBR_OK);
  return t;
}
static bool same(const gbr_tuning& a, const gbr_tuning& b) { return std::memcmp(&a, &b, sizeof a) == 0; }

static void run(uint32_t scenes, int w, int h, uint32_t draws) {
  const cudaStream_t stream = fake::stream(false);
  Renderer* r = fake::renderer(scenes, w, h, draws);
  const gbr_tuning chosen = get(r);
  int threads = 0;
  RasterParams last{};
  fake::on_raster = [&](const RasterParams& p, int t, uint32_t, size_t) {
    threads = t;
    last = p;
  };
  CHECK(r->draw(stream, GBR_DRAW_PER_SCENE, false) == GBR_OK);
  CHECK(same(get(r), chosen));
  CHECK(threads == chosen.threads && last.small_area == chosen.small_area &&
        last.region_w == chosen.plain_region_width && last.region_h == chosen.plain_region_height);

  // One field, before and after the first draw: the same shape otherwise.
  Renderer* early = fake::renderer(scenes, w, h, draws);
  gbr_tuning off{};
  CHECK(early->set_tuning(off, 1u << 7) == GBR_OK && r->set_tuning(off, 1u << 7) == GBR_OK);
  gbr_tuning want = chosen;
  want.occlusion_culling = 0;
  CHECK(same(get(early), want) && same(get(r), want));
  CHECK(early->draw(stream, GBR_DRAW_BATCHED, false) == GBR_OK && r->draw(stream, GBR_DRAW_BATCHED, false) == GBR_OK);
  CHECK(threads == chosen.threads && last.occlusion == 0);
  CHECK(same(get(early), want) && same(get(r), want));
  delete early;

  // A region of one's own, and threads of one's own.
  gbr_tuning t{};
  t.region_width = t.region_height = 128;
  CHECK(r->set_tuning(t, 2u | 4u) == GBR_OK);
  want.region_width = want.region_height = 128;
  want.threads = 1024;  // two such z-buffers do not fit an SM
  want.ctas_per_sm = 1;
  gbr_tuning now = get(r);
  CHECK(now.region_width == 128 && now.region_height == 128 && now.threads == 1024 && now.ctas_per_sm == 1);
  CHECK(r->draw(stream, GBR_DRAW_BATCHED, false) == GBR_OK && threads == 1024);
  t.plain_region_height = 1024;
  CHECK(r->set_tuning(t, 1u << 6) == GBR_OK);
  now = get(r);
  CHECK(now.plain_region_height == 1024 && now.plain_region_width >= 4);
  CHECK(r->draw(stream, GBR_DRAW_PER_SCENE, false) == GBR_OK && last.region_h == 1024);
  t.plain_region_width = 64;
  CHECK(r->set_tuning(t, 1u << 5) == GBR_ERROR_INVALID_ARGUMENT);  // 64 x 1024
  CHECK(same(get(r), now));
  t.threads = 100;
  CHECK(r->set_tuning(t, 1u) == GBR_ERROR_INVALID_ARGUMENT);
  CHECK(same(get(r), now));
  // All of them: as given.
  const gbr_tuning all{256, 32, 32, 9, 3, 8, 24, 1, 50};
  CHECK(r->set_tuning(all) == GBR_OK && same(get(r), all));
  CHECK(r->draw(stream, GBR_DRAW_PER_SCENE, false) == GBR_OK && threads == 256 && last.region_w == 8);
  CHECK(same(get(r), all));
  delete r;
}

int main() {
  run(1, 128, 128, 3);
  run(48, 160, 120, 200);
  run(600, 128, 128, 20);
  return fake::finish();
}
