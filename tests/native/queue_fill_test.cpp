// The queue's share of the threads: every step from 25 to 68 and from 76 to 100 %
// is a launch of its own, and a full queue fits two CTAs of the default shape.
#include <cuda_runtime.h>

#include <cstdio>

#include "kernels.h"
#include "records.h"

using namespace gbr;

int main() {
  int failures = 0;
  for (int threads : {256, 512, 1024}) {
    uint32_t last = 0;
    for (int percent = 25; percent <= 100; ++percent) {
      const uint32_t at = raster_flush_at(threads, percent), cap = raster_queue_cap(threads, percent);
      const bool full = percent >= 69 && percent <= 75;
      if (at < 1 || at > cap || cap > uint32_t(threads) || (full ? at != cap : at <= last)) {
        std::fprintf(stderr, "%d threads, %d %%: flush at %u of %u\n", threads, percent, at, cap);
        ++failures;
      }
      last = at;
    }
    if (raster_flush_at(threads, 100) != uint32_t(threads)) ++failures;
  }
  const size_t one = raster_smem_bytes(512, 128, 64, 0, raster_queue_cap(512, 100));
  if (2 * (one + 2048) > 233472) {
    std::fprintf(stderr, "%zu bytes\n", one);
    ++failures;
  }
  if (failures) return 1;
  std::printf("ok\n");
  return 0;
}
