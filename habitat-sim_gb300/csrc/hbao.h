// Horizon-based ambient occlusion kernels and their host-side parameters
// (shared by the renderer's gbr_hbao_draw and the standalone gbr_hbao_apply).
#pragma once
#include <cuda_runtime.h>

#include <cstdint>
#include <string>

#include "../../include/gbr_hbao.h"

namespace gbr {

// One image: its rectangle in the planes, projection info and radius.
struct HbaoScene {
  long long offset;  // element index of pixel (0, 0) (bottom-left)
  long long pitch;   // elements per row
  int w, h;
  float pi[4];       // view position = ((u, v) * pi.xy + pi.zw) * z (z = 1 if orthographic)
  float radius_to_screen;
  float far_plane;   // depth given to background pixels (linear depth 0)
  int ortho;
  int block0, blur0; // first block of the scene in the AO and in the blur grid
  int qw, qh;        // quarter resolution of the cache-aware algorithm: ceil(w / 4) x ceil(h / 4)
  float inv_qw, inv_qh;  // 1 / qw, 1 / qh
  float inv_w, inv_h;    // 1 / w, 1 / h
  int fits;          // w, h <= 65536 and h * pitch < 2^31: 32-bit texel arithmetic is exact
};

// One block of the AO grid covers kAoTile x kAoTile pixels of a scene, one of
// the blur grid kBlurTile x kBlurTile.
constexpr int kAoTile = 16, kBlurTile = 32;
inline long long hbao_blocks(int w, int h, int tile) {
  return ((w + tile - 1LL) / tile) * ((h + tile - 1LL) / tile);
}

// How far the AO kernel's estimated sum of 32 samples (reciprocal root by
// rsqrt.approx, fused sums) may be from the specification's, both in single
// precision from the same N, V, radius and bias; u = 2^-24, n = |N|.
//   Specification: N.V off by 3 u n |V| (a product and two sums, Cauchy-Schwarz),
//   |V| by 2.5 u (|V|^2 by 3 u, the root halves it and rounds), the quotient
//   rounds: 6.5 u n.  Less the bias: u.  The falloff (the product of |V|^2 by
//   4 u, the sum 1 u) 5 u, the product of both u: (6.5 n + 7) u.
//   Estimate: N.V 3 u n |V|, the reciprocal root 2^-22.9 < 2.15 u and half of
//   |V|^2's 3 u, the product u: 7.65 u n.  The bias u, the falloff 4 u (fused);
//   the last product is exact inside the sum: (7.65 n + 5) u.
// Both factors are clamped to [0, 1], which does not add.  The cache-aware normal
// comes from bytes: each component within 1/255, so n <= 1 + sqrt(3) / 255.
// The sums of non-negative terms round 31 and 32 times, by u of the sum each.
constexpr double kAoUnit = 1.0 / 16777216.0, kAoNormal = 1.0 + 1.7320509 / 255.0;
constexpr double kAoSampleError = (14.15 * kAoNormal + 12.0) * kAoUnit;
constexpr float kAoSumError = 5.1e-5f, kAoSumRelative = 5e-6f;
static_assert(32.0 * kAoSampleError < 0.99 * kAoSumError && 63.0 * kAoUnit < 0.99 * kAoSumRelative,
              "the estimate's bound holds every rounding (and those of the bound itself)");
// poly_pow(a, e) for a in [0, 1] is off a^e by less than half of this, at
// whichever e (measured, tests/test_hbao_bound_host.py).
constexpr float kAoPowSlack = 5e-7f, kAoPowSlackPerExponent = 3e-7f;

struct HbaoParams {
  float neg_inv_r2, bias, bias2, ao_scale, pow_exp, sharpness;  // bias2: see hbao_ao_kernel
  int no_blur;
  int special;       // AO and view depth kept as two halves per pixel, blurred with that depth
  int cache_aware;   // the deinterleaved algorithm
  float jitter[64];  // 4 x 4 texels of (cos, sin, start offset, 0), 16-bit snorm (classic)
  float jitter_f[64];  // the same, unquantized (cache-aware: one per deinterleaved layer)
  float dirs[16];    // 8 unit directions (cos, sin)
};

void hbao_jitter_unquantized(float out[64]);
// Validates the configuration and fills the per-call constants.
bool hbao_params(const gbr_hbao_config& c, HbaoParams& p, std::string& err);
// Per-image constants from a column-major projection (Hbao.cpp:761-786, 874-895).
HbaoScene hbao_scene(const float* projection, int w, int h, long long offset, long long pitch,
                     float radius);
// Bytes per pixel of the intermediate plane: an 8-bit AO, or with the special
// blur an (AO, view depth) pair of halves.
inline int hbao_plane_bytes(const HbaoParams& p) { return p.special ? 4 : 1; }
// Two launches on `stream`: AO (into q, or straight into colour without
// blur), then both blur passes and the colour multiply.  q has the colour
// plane's layout, hbao_plane_bytes(p) per pixel.  The scenes are read from
// device memory, or with count 1 and d_scenes null from `one`; ao_blocks and
// blur_blocks are the sums of hbao_blocks() over them.
cudaError_t hbao_launch(const HbaoScene* d_scenes, const HbaoScene& one, int count, int ao_blocks,
                        int blur_blocks, const float* depth, uint32_t* color, void* q, const HbaoParams& p,
                        cudaStream_t stream);

}  // namespace gbr
