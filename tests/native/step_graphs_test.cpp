// Captured graphs while scenes come and go, as a request server's do: each form
// of the step is captured once per staging slot and never again, and every step
// is launched with a z-buffer that holds its items, over the list that it reads.
#include "renderer.cpp"

#include <random>

#include "fake_cuda.h"

using namespace gbr;

static void run(uint32_t n, int w, int h, const gbr_tuning* tuning) {
  Renderer* r = fake::renderer(n, w, h);
  if (tuning) CHECK(r->set_tuning(*tuning) == GBR_OK);
  const cudaStream_t stream = fake::stream(false);
  uint32_t on = 0;
  bool ordered = false;
  uint32_t launched = 0;
  fake::on_order = [&](const RasterParams& p, uint32_t, uint32_t*) {
    ordered = true;
    // The kernel sorts this list into the one behind it.
    WorkItem* list = const_cast<WorkItem*>(p.items);
    std::copy(list, list + *p.item_count_dev, list + p.item_count);
  };
  fake::on_raster = [&](const RasterParams& p, int threads, uint32_t, size_t smem) {
    ++launched;
    CHECK(smem == raster_smem_bytes(threads, p.region_w, p.region_h, p.prefix_cap, p.queue_cap));
    CHECK((p.item_base != 0) == ordered);
    const uint32_t count = *p.item_count_dev;
    CHECK(count <= p.item_count);
    uint64_t pixels = 0;
    for (uint32_t i = 0; i < count; ++i) {
      const WorkItem& it = p.items[p.item_base + i];
      CHECK(it.w * it.h <= p.region_w * p.region_h);
      CHECK(ordered || (it.w <= p.region_w && it.h <= p.region_h));
      pixels += uint64_t(it.w) * it.h;
    }
    CHECK(pixels == uint64_t(on) * uint64_t(w) * uint64_t(h));
    ordered = false;
  };
  std::mt19937 rng(n);
  const int before = fake::captures;
  int warm = 0;
  for (int step = 0; step < 120; ++step) {
    if (step == 80) warm = fake::captures;
    // Light, changing load, with a full step now and then.
    const uint32_t want = step % 10 == 9 ? n : 1 + rng() % (step % 2 ? n : std::min(n, 24u));
    for (uint32_t s = 0; s < n; ++s) CHECK(r->set_enabled(s, s < want) == GBR_OK);
    on = want;
    CHECK(r->draw(stream, GBR_DRAW_BATCHED, true) == GBR_OK);
    gbr_draw_stats st;
    CHECK(r->last_stats(&st) == GBR_OK && (st.kernel_launches == 2 || st.kernel_launches == 3));
  }
  CHECK(launched == 120);
  CHECK(fake::captures - before <= 6);
  CHECK(fake::captures == warm);
  delete r;
}

int main() {
  run(320, 128, 128, nullptr);
  run(64, 64, 64, nullptr);
  run(20, 256, 256, nullptr);
  run(3, 100, 37, nullptr);
  gbr_tuning t{1024, 128, 128, 1, 1, 16, 32, 1, 75};
  run(200, 128, 128, &t);
  return fake::finish();
}
