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
  bool resources = true;
  fake::on_raster = [&](const RasterParams& p, int, uint32_t, size_t) {
    items = *p.item_count_dev;
    // What the library and the caller added before: texels, indices, boxes.
    resources = p.texels[0] == 0xffffffffu && p.boxes[0].hi[0] == 1.0f;
    for (uint32_t i = 0; i < 3; ++i) resources = resources && p.indices[i] == i;
  };
  for (int round = 0; round < 2; ++round) {
    CHECK(r->draw(stream, GBR_DRAW_BATCHED, false) == GBR_OK);
    CHECK(scenes_seen == 200);
    CHECK(resources);
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
  // More of everything: the buffers grow, and what they held is there.
  for (int k = 0; k < 40; ++k) {
    const float pos[9] = {0, 0, -1, 1, 0, -1, 0, 1, -1};
    const uint32_t idx[3] = {2, 1, 0};
    gbr_mesh_data m{};
    m.vertex_count = m.index_count = 3;
    m.positions = pos;
    m.indices = idx;
    uint32_t id;
    CHECK(r->add_mesh(m, &id) == GBR_OK);
    gbr_mesh_view v{};
    v.mesh = id;
    v.index_count = 3;
    CHECK(r->add_template(("t" + std::to_string(k)).c_str(), 1, &v) == GBR_OK);
    const uint8_t texel[4] = {1, 2, 3, 4};
    gbr_texture_data t{1, 1, 1, texel, 0, 0, 0};
    CHECK(r->add_texture(t, &id) == GBR_OK);
    CHECK(r->draw(stream, GBR_DRAW_BATCHED, false) == GBR_OK);
    CHECK(resources);
  }
  delete r;
  return fake::finish();
}
