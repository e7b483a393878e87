// Draws on a non-blocking stream while the legacy default stream is busy: what
// a draw that rebuilds the scene tables writes to device memory is in place
// before its kernels run, and nothing is written over it later.
#include "renderer.cpp"

#include "fake_cuda.h"

using namespace gbr;

int main() {
  Renderer* r = fake::renderer(200, 128, 128);
  const cudaStream_t stream = fake::stream(false);
  uint32_t items = 0, scenes_seen = 0;
  uint32_t* done_word = nullptr;
  uint32_t* status = nullptr;
  fake::on_prepare = [&](const PrepareParams& p, uint32_t n) {
    scenes_seen = 0;
    for (uint32_t s = 0; s < n; ++s) scenes_seen += p.scenes[s].width == 128 && p.scenes[s].draw_count == 1;
    status = p.status;
  };
  fake::on_order = [&](const RasterParams&, uint32_t, uint32_t* done) { done_word = done; };
  fake::on_raster = [&](const RasterParams& p, int, uint32_t, size_t) { items = *p.item_count_dev; };
  for (int round = 0; round < 2; ++round) {
    CHECK(r->draw(stream, GBR_DRAW_BATCHED, false) == GBR_OK);
    CHECK(scenes_seen == 200);
    CHECK(items >= 400 && done_word && status);
    if (!done_word || !status) return 1;
    const uint32_t drawn = items;
    // The kernels are under way when the legacy stream gets to its work.
    *done_word = 5;
    *status = kStatusBadNode;
    fake::run_legacy();
    CHECK(*done_word == 5);
    CHECK(*status == kStatusBadNode);
    *done_word = 0;
    *status = 0;
    CHECK(r->draw(stream, GBR_DRAW_BATCHED, false) == GBR_OK);
    CHECK(items == drawn);
    // A bad record: reported once, then the tables are built again.
    *status = kStatusBadNode;
    gbr_draw_stats st;
    CHECK(r->last_stats(&st) == GBR_ERROR_DEVICE);
    CHECK(*status == 0);
  }
  delete r;
  return fake::finish();
}
