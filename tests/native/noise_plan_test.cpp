// How batches of images are cut for the noise kernel: every pixel exactly once;
// a block's threads are at least half busy, and with tables no block has much
// more to do than the mean, whatever the images' size.
#include <cmath>
#include <cstdio>
#include <random>
#include <vector>

#include "noise_plan.h"

using namespace gbr;

static int failures = 0;
#define CHECK(c, w, h, n)                                                                  \
  do {                                                                                     \
    if (!(c)) {                                                                            \
      std::fprintf(stderr, "%s:%d: %s (%u of %u x %u)\n", __FILE__, __LINE__, #c, n, w, h); \
      ++failures;                                                                          \
    }                                                                                      \
  } while (0)

static void check(uint32_t w, uint32_t h, uint32_t n) {
  const uint32_t sms = 152;
  const NoisePlan p = noise_plan(w, h, n, sms);
  const uint32_t threads = (p.form >= NoisePlan::kTable) ? kNoiseTableThreads : kNoisePlainThreads;
  const uint64_t pixels = uint64_t(w) * h;
  CHECK(p.chunk % threads == 0 && p.grid >= 1 && p.grid <= p.units, w, h, n);
  std::vector<uint64_t> passes(p.grid, 0);
  uint64_t covered = 0, all = 0;
  CHECK((p.form == NoisePlan::kPacked) == (p.pack > 1), w, h, n);
  CHECK(p.pack == 1 || (p.chunks == 1 && p.pack * pixels <= threads), w, h, n);
  for (uint64_t u = 0; u < p.units; ++u) {
    const uint64_t first = (p.form == NoisePlan::kTableSpread ? u / n : u % p.chunks) * p.chunk;
    const uint64_t images = std::min<uint64_t>(p.pack, uint64_t(n) * p.chunks - u * p.pack);
    CHECK(first < pixels && u * p.pack < uint64_t(n) * p.chunks, w, h, n);
    const uint64_t here = images * std::min<uint64_t>(p.chunk, pixels - first), k = (here + threads - 1) / threads;
    covered += here;
    passes[u % p.grid] += k;
    all += k;
  }
  CHECK(covered == pixels * n, w, h, n);
  // A block's threads are at least half busy (but for a last unit).
  CHECK(2 * covered >= (all - 1) * threads, w, h, n);
  if (!(p.form >= NoisePlan::kTable)) return;
  uint64_t most = 0;
  for (uint64_t b : passes) most = std::max(most, b);
  // The mean, one pass of imbalance per chunk position and a last unit.
  CHECK(double(most) <= 1.25 * double(all) / p.grid + 2.0 * p.chunk / threads, w, h, n);
}

int main() {
  const uint32_t sizes[][3] = {{1, 1, 1u << 21},  {8, 8, 1u << 15},    {20, 20, 10496}, {24, 24, 7296},  {32, 32, 4096},
                               {36, 33, 1792},    {60, 80, 1760},      {60, 80, 896},   {64, 64, 1024},  {128, 128, 1024},
                               {4096, 4096, 1},   {1, 4095, 260},      {640, 480, 30},  {33, 31, 2},     {1, 1, 1}};
  for (const auto& s : sizes) check(s[0], s[1], s[2]);
  std::mt19937 rng(3);
  for (int k = 0; k < 200; ++k) {
    const uint32_t w = 1 + rng() % 200, h = 1 + rng() % 200;
    check(w, h, 1 + uint32_t((uint64_t(1) << (18 + rng() % 6)) / (uint64_t(w) * h)));
  }
  if (failures) return 1;
  std::printf("ok\n");
  return 0;
}
