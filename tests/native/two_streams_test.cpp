// Draws of one renderer on different streams follow one another; a draw in the
// caller's capture waits for nothing outside it.
#include "renderer.cpp"

#include "fake_cuda.h"

using namespace gbr;

int main() {
  Renderer* r = fake::renderer(200, 128, 128);
  const cudaStream_t a = fake::stream(false), b = fake::stream(false);
  CHECK(r->draw(a, GBR_DRAW_BATCHED, false) == GBR_OK);
  CHECK(r->draw(a, GBR_DRAW_BATCHED, true) == GBR_OK);
  CHECK(fake::waits.empty());
  cudaStream_t last = a;
  for (const uint32_t mode : {GBR_DRAW_BATCHED, GBR_DRAW_PER_SCENE})
    for (const cudaStream_t s : {b, a, cudaStream_t(nullptr), b, a}) {
      fake::waits.clear();
      CHECK(r->draw(s, mode, false) == GBR_OK);
      CHECK(fake::waits.size() == (s != last ? 1u : 0u));
      if (!fake::waits.empty()) CHECK(fake::waits[0].first == s && fake::waits[0].second == last);
      last = s;
      fake::waits.clear();
      CHECK(r->draw(s, mode, false) == GBR_OK);
      CHECK(fake::waits.empty());
    }
  // The caller's capture of another stream.
  fake::waits.clear();
  cudaGraph_t g;
  CHECK(cudaStreamBeginCapture(b, cudaStreamCaptureModeRelaxed) == cudaSuccess);
  CHECK(r->draw(b, GBR_DRAW_BATCHED, false) == GBR_OK);
  CHECK(cudaStreamEndCapture(b, &g) == cudaSuccess);
  CHECK(fake::waits.empty());
  cudaGraphDestroy(g);
  delete r;
  return fake::finish();
}
