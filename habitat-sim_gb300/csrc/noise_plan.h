// How a batch of depth images is cut for the noise kernel (noise.cu): pure
// host arithmetic, no CUDA.
#pragma once

#include <algorithm>
#include <cstdint>

namespace gbr {

// With tables a block is large and fills shared memory first; without, small.
constexpr uint32_t kNoiseTableThreads = 1024, kNoisePlainThreads = 256;
constexpr uint64_t kNoiseTablePixels = 1u << 20;

// Units of the launch, of `chunk` pixels each (fewer at an image's end); block b
// takes units b, b + grid, ...
//   kPlain, kTable  unit u: chunk u % chunks of image u / chunks
//   kTableSpread    unit u: chunk u / count of image u % count
//   kPacked         unit u: `pack` whole images from pack * u on
struct NoisePlan {
  enum Form { kPlain, kPacked, kTable, kTableSpread } form;
  uint32_t chunk;   // a multiple of the block's threads
  uint32_t chunks;  // per image
  uint32_t pack;    // images per unit
  uint64_t units;
  uint32_t grid;
};

// Tables where they pay: in batches of 1 M pixels (64 images of 128 x 128: 14.4
// us against 16.5 without; 32: 11.7 against 10.3) whose images fill half of the
// blocks' threads (4 M pixels as 24 x 24 images: 55 us against 62 without; 20 x
// 20: 68 against 62; 1 x 1: 15.9 ms against 1.5), the more the smaller the batch
// (1 M pixels as 33 x 33 images: 20.5 against 18.5; as 48 x 37: 16.4 against
// 18.4).  Chunks of four pixels per thread where that leaves every block several.
// Where an image ends in a shorter chunk the units go chunk by chunk over all
// images, so that the short ones are spread over the blocks: image by image, with
// two chunks each and an even grid, one half of the blocks got all of them (1760
// images of 80 x 60: 113 us, 107 without tables, 72 now).
// Without tables, images of at most half a block's threads share a block: one
// image to a block leaves its other threads idle (4 M pixels as 8 x 8 images: 62
// us instead of 82, as 1 x 1: 49 instead of 1530).
inline NoisePlan noise_plan(uint32_t tw, uint32_t th, uint32_t count, uint32_t sms) {
  const uint64_t pixels = uint64_t(tw) * th, total = pixels * count;
  const uint64_t threads = (pixels + kNoiseTableThreads - 1) / kNoiseTableThreads * kNoiseTableThreads;
  const bool table = total >= kNoiseTablePixels && 2 * pixels >= kNoiseTableThreads &&
                     4.0 * double(total) * double(pixels) >= 3.0 * double(kNoiseTablePixels) * double(threads);
  NoisePlan p;
  p.pack = table ? 1 : std::max<uint32_t>(1, uint32_t(kNoisePlainThreads / std::min<uint64_t>(pixels, kNoisePlainThreads)));
  p.chunk = !table ? kNoisePlainThreads : kNoiseTableThreads * (total >= 4 * kNoiseTablePixels ? 4 : 1);
  p.chunks = uint32_t((pixels + p.chunk - 1) / p.chunk);
  p.form = table ? (pixels % p.chunk == 0 ? NoisePlan::kTable : NoisePlan::kTableSpread)
                 : (p.pack > 1 ? NoisePlan::kPacked : NoisePlan::kPlain);
  p.units = (uint64_t(p.chunks) * count + p.pack - 1) / p.pack;
  p.grid = uint32_t(std::min<uint64_t>(p.units, table ? 2 * sms : 0x7fffffffu));
  return p;
}

}  // namespace gbr
