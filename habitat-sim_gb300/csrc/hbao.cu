// Horizon-based ambient occlusion, classic algorithm (declared in
// include/gbr_hbao.h; restating src/esp/gfx_batch/Hbao.cpp:595-935 and the
// shaders src/shaders/gfx_batch/hbao/hbao.frag, bilateralblur.frag).
//
// Per pixel (x, y) of a w x h image with linear depth L (0 -> far plane),
// u = (x + 0.5) / w, v = (y + 0.5) / h:
//   P = ((u, v) * pi.xy + pi.zw) * z, z)         view position (z = 1 in x, y if orthographic)
//   N = -normalize(cross(dx, dy)), dx / dy the shorter of the forward and
//       backward differences to the neighbouring pixels (clamped at edges)
//   R = radius_to_screen / z pixels, step = R / 5, jitter J = table[y & 3][x & 3]
//   for 8 directions d rotated by J.xy, 4 steps from J.z * step + 1 pixels:
//       S = the view position at P's pixel + rint(ray * d) (clamped texel,
//           unclamped coordinates), V = S - P,
//       AO += clamp(N.V / |V| - bias, 0, 1) * clamp(1 - |V|^2 / r^2, 0, 1)
//   ao = clamp(1 - 2 AO / (1 - bias) / 32, 0, 1) ^ intensity, stored as unorm8
// then a 7-tap blur along x, stored as unorm8, along y, each tap weighted
// exp2(-t^2 / 4.5 - ((L_t - L_c) sharpness)^2), and colour rgb *= ao.
//
// pow and exp2 are evaluated by the polynomials below (exp2: Taylor series of
// 2^f on [0, 1) to degree 9 and exact scaling; log2: atanh series of the
// mantissa normalised to [sqrt(1/2), sqrt(2))), every operation one float
// rounding, so the result is a pure function of the inputs that the
// oracle reproduces bit for bit.  GLSL leaves pow/exp2 precision to the
// driver; this fixes it.
#include "hbao.h"

#include <cuda_fp16.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <random>
#include <vector>

namespace gbr {
void set_last_error(const std::string& msg);

namespace {

// Two floats in a register pair: an addition of pairs is one instruction and
// rounds each half as the scalar one does.  Products are left to two scalar
// instructions, also where a pair's would do: the assembler contracts a pair's
// multiplication and addition into one fused operation whatever their rounding
// modifiers and flags say, and a fused result is another number.  (fma2 is for where
// that is wanted.)
struct F2 {
  unsigned long long v;
};
__device__ __forceinline__ F2 f2(float lo, float hi) {
  F2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r.v) : "f"(lo), "f"(hi));
  return r;
}
__device__ __forceinline__ F2 f2(float a) { return f2(a, a); }
__device__ __forceinline__ float2 split(F2 a) {
  float2 r;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(a.v));
  return r;
}
__device__ __forceinline__ F2 add2(F2 a, F2 b) {
  F2 r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
  return r;
}
__device__ __forceinline__ F2 mul2(F2 a, F2 b) {
  const float2 x = split(a), y = split(b);
  return f2(__fmul_rn(x.x, y.x), __fmul_rn(x.y, y.y));
}
__device__ __forceinline__ F2 fma2(F2 a, F2 b, F2 c) {
  F2 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r.v) : "l"(a.v), "l"(b.v), "l"(c.v));
  return r;
}

__device__ __forceinline__ float poly_exp2(float x) {
  if (x < -149.0f) return 0.0f;
  const float n = floorf(x);
  const float f = __fsub_rn(x, n);
  float p = 1.0178086284895471e-07f;
  p = __fadd_rn(__fmul_rn(p, f), 1.3215486660556053e-06f);
  p = __fadd_rn(__fmul_rn(p, f), 1.5252733646775596e-05f);
  p = __fadd_rn(__fmul_rn(p, f), 0.0001540352968731895f);
  p = __fadd_rn(__fmul_rn(p, f), 0.0013333557872101665f);
  p = __fadd_rn(__fmul_rn(p, f), 0.009618128649890423f);
  p = __fadd_rn(__fmul_rn(p, f), 0.05550410971045494f);
  p = __fadd_rn(__fmul_rn(p, f), 0.24022650718688965f);
  p = __fadd_rn(__fmul_rn(p, f), 0.6931471824645996f);
  p = __fadd_rn(__fmul_rn(p, f), 1.0f);
  // p 2^n for n in [-149, 0] (every caller's x is at most 0) in two factors:
  // the first product is exact, the second rounds once, into the denormals.
  const int k = int(n), k1 = max(k, -126);
  return __fmul_rn(__fmul_rn(p, __int_as_float((k1 + 127) << 23)), __int_as_float((k - k1 + 127) << 23));
}

// poly_exp2 of both halves.
__device__ __forceinline__ float2 poly_exp2(F2 x2) {
  const float2 x = split(x2);
  const float n0 = floorf(x.x), n1 = floorf(x.y);
  const F2 f = add2(x2, f2(-n0, -n1));
  F2 p = f2(1.0178086284895471e-07f);
  p = add2(mul2(p, f), f2(1.3215486660556053e-06f));
  p = add2(mul2(p, f), f2(1.5252733646775596e-05f));
  p = add2(mul2(p, f), f2(0.0001540352968731895f));
  p = add2(mul2(p, f), f2(0.0013333557872101665f));
  p = add2(mul2(p, f), f2(0.009618128649890423f));
  p = add2(mul2(p, f), f2(0.05550410971045494f));
  p = add2(mul2(p, f), f2(0.24022650718688965f));
  p = add2(mul2(p, f), f2(0.6931471824645996f));
  p = add2(mul2(p, f), f2(1.0f));
  const int k0 = int(n0), k1 = int(n1), m0 = max(k0, -126), m1 = max(k1, -126);
  p = mul2(p, f2(__int_as_float((m0 + 127) << 23), __int_as_float((m1 + 127) << 23)));
  const float2 r = split(mul2(p, f2(__int_as_float((k0 - m0 + 127) << 23), __int_as_float((k1 - m1 + 127) << 23))));
  return make_float2(x.x < -149.0f ? 0.0f : r.x, x.y < -149.0f ? 0.0f : r.y);
}

__device__ __forceinline__ float poly_log2(float x) {
  int e;
  float m = frexpf(x, &e);
  if (m < 0.7071067690849304f) {
    m = __fmul_rn(m, 2.0f);
    e -= 1;
  }
  const float t = __fdiv_rn(__fsub_rn(m, 1.0f), __fadd_rn(m, 1.0f));
  const float t2 = __fmul_rn(t, t);
  float q = 0.1111111119389534f;
  q = __fadd_rn(__fmul_rn(q, t2), 0.1428571492433548f);
  q = __fadd_rn(__fmul_rn(q, t2), 0.20000000298023224f);
  q = __fadd_rn(__fmul_rn(q, t2), 0.3333333432674408f);
  q = __fadd_rn(__fmul_rn(q, t2), 1.0f);
  return __fadd_rn(float(e), __fmul_rn(__fmul_rn(t, q), 2.885390043258667f));
}

__device__ __forceinline__ float poly_pow(float a, float e) {
  if (!(a > 0.0f)) return e == 0.0f ? 1.0f : 0.0f;
  return poly_exp2(__fmul_rn(e, poly_log2(a)));
}

// Relative error at most 2^-22.9.
__device__ __forceinline__ float rsqrt_approx(float a) {
  float r;
  asm("rsqrt.approx.f32 %0, %1;" : "=f"(r) : "f"(a));
  return r;
}

__device__ __forceinline__ float clamp01(float v) { return fminf(fmaxf(v, 0.0f), 1.0f); }

__device__ __forceinline__ float3 f3(float x, float y, float z) { return make_float3(x, y, z); }
__device__ __forceinline__ float3 sub(float3 a, float3 b) {
  return f3(__fsub_rn(a.x, b.x), __fsub_rn(a.y, b.y), __fsub_rn(a.z, b.z));
}
__device__ __forceinline__ float dot3(float3 a, float3 b) {
  return __fadd_rn(__fadd_rn(__fmul_rn(a.x, b.x), __fmul_rn(a.y, b.y)), __fmul_rn(a.z, b.z));
}
__device__ __forceinline__ float3 cross3(float3 a, float3 b) {
  return f3(__fsub_rn(__fmul_rn(a.y, b.z), __fmul_rn(a.z, b.y)),
            __fsub_rn(__fmul_rn(a.z, b.x), __fmul_rn(a.x, b.z)),
            __fsub_rn(__fmul_rn(a.x, b.y), __fmul_rn(a.y, b.x)));
}

__device__ __forceinline__ float depth_at(const HbaoScene& s, const float* __restrict__ depth, int tx, int ty) {
  tx = min(max(tx, 0), s.w - 1);
  ty = min(max(ty, 0), s.h - 1);
  const float z = __ldg(depth + s.offset + (long long)ty * s.pitch + tx);
  return z == 0.0f ? s.far_plane : z;
}

__device__ __forceinline__ float3 view_pos(const HbaoScene& s, float u, float v, float z) {
  const float k = s.ortho ? 1.0f : z;
  return f3(__fmul_rn(__fadd_rn(__fmul_rn(u, s.pi[0]), s.pi[2]), k),
            __fmul_rn(__fadd_rn(__fmul_rn(v, s.pi[1]), s.pi[3]), k), z);
}

__device__ __forceinline__ float3 min_diff(float3 p, float3 pr, float3 pl) {
  const float3 v1 = sub(pr, p), v2 = sub(p, pl);
  return dot3(v1, v1) < dot3(v2, v2) ? v1 : v2;
}

__device__ __forceinline__ uint8_t unorm8(float v) {
  return uint8_t(__fadd_rn(__fmul_rn(clamp01(v), 255.0f), 0.5f));
}

// v / 255 correctly rounded for a byte v: 1/255 as the sum of two floats, one
// multiply and one fused multiply-add (Brisebarre and Muller, "Correctly
// rounded multiplication by arbitrary precision constants", IEEE Trans.
// Computers 57(2), 2008; checked for all 256 v in exact rational arithmetic).
__device__ __forceinline__ float byte_unit(uint32_t v) {
  const float f = __fsub_rn(__uint_as_float(0x4b000000u | v), 8388608.0f);
  return __fmaf_rn(f, 0x1.010102p-8f, __fmul_rn(f, -0x1.fdfdfep-33f));
}

__device__ __forceinline__ uint32_t modulate(uint32_t c, float ao) {
  uint32_t out = c & 0xFF000000u;  // alpha: blend factor one
  for (int ch = 0; ch < 3; ++ch) {
    const float v = __fmul_rn(byte_unit((c >> (8 * ch)) & 0xFFu), ao);
    out |= uint32_t(unorm8(v)) << (8 * ch);
  }
  return out;
}

// The scene of this block, by a binary search of thread 0, and the block's
// index among the scene's.  First: the scenes' first blocks (block0 or blur0).
template <int HbaoScene::*First>
__device__ __forceinline__ int scene_of_block(const HbaoScene* scenes, int count, int* local) {
  __shared__ int s_si, s_local;
  if (threadIdx.x == 0) {
    int lo = 0, hi = count;  // scenes[lo].*First <= blockIdx.x < scenes[hi].*First
    while (hi - lo > 1) {
      const int mid = (lo + hi) >> 1;
      if (scenes[mid].*First <= int(blockIdx.x))
        lo = mid;
      else
        hi = mid;
    }
    s_si = lo;
    s_local = int(blockIdx.x) - scenes[lo].*First;
  }
  __syncthreads();
  *local = s_local;
  return s_si;
}

__device__ __forceinline__ float3 reconstruct_normal(const HbaoScene& s, const float* __restrict__ depth, int x, int y,
                                                     float u, float v, float inv_w, float inv_h, float3 P,
                                                     float& inv_len) {
  const float3 pr = view_pos(s, __fadd_rn(u, inv_w), v, depth_at(s, depth, x + 1, y));
  const float3 pl = view_pos(s, __fadd_rn(u, -inv_w), v, depth_at(s, depth, x - 1, y));
  const float3 pt = view_pos(s, u, __fadd_rn(v, inv_h), depth_at(s, depth, x, y + 1));
  const float3 pb = view_pos(s, u, __fadd_rn(v, -inv_h), depth_at(s, depth, x, y - 1));
  const float3 c = cross3(min_diff(P, pr, pl), min_diff(P, pt, pb));
  inv_len = __fdiv_rn(1.0f, __fsqrt_rn(dot3(c, c)));
  return c;
}

// Depth of the cache-aware sample: texel (tqx, tqy) of deinterleaved layer
// (ox, oy), i.e. full-resolution pixel (4 tqx + ox, 4 tqy + oy); texels of
// the quarter-resolution layer that fall beyond the image read as the far plane.
__device__ __forceinline__ float layer_depth(const HbaoScene& s, const float* __restrict__ depth, int tqx, int tqy,
                                             int ox, int oy) {
  tqx = min(max(tqx, 0), s.qw - 1);
  tqy = min(max(tqy, 0), s.qh - 1);
  const int fx = 4 * tqx + ox, fy = 4 * tqy + oy;
  if (fx >= s.w || fy >= s.h) return s.far_plane;
  const float z = __ldg(depth + s.offset + (long long)fy * s.pitch + fx);
  return z == 0.0f ? s.far_plane : z;
}

__device__ __forceinline__ uint32_t pack_half2(float a, float b) {
  return uint32_t(__half_as_ushort(__float2half_rn(a))) | (uint32_t(__half_as_ushort(__float2half_rn(b))) << 16);
}
__device__ __forceinline__ float half_lo(uint32_t v) { return __half2float(__ushort_as_half((unsigned short)(v & 0xFFFFu))); }
__device__ __forceinline__ float half_hi(uint32_t v) { return __half2float(__ushort_as_half((unsigned short)(v >> 16))); }

// What the samples of one pixel need.
struct AoPixel {
  float3 P, N;
  float u, v, su_scale, sv_scale;
  int x, y;
};

// Adds a sample's AO: squared distance vv, N.V nv, and the falloff at vv.
__device__ __forceinline__ float ao_add(const HbaoParams& p, float ao, float vv, float nv, float fall) {
  // Most samples add exactly nothing and leave before the square root and the
  // division: beyond the radius (fall <= 0 or not a number), behind the
  // tangent plane, or below the bias: N.V / |V| < bias, decided on squares
  // with a margin (bias2 = bias^2 (1 - 1e-5)) far above the roundings of
  // either side, for |V| where the squares are normal numbers.
  if (!(fall > 0.0f) || !(nv > 0.0f) || (vv > 1e-20f && __fmul_rn(nv, nv) < __fmul_rn(p.bias2, vv))) return ao;
  const float ndotv = __fdiv_rn(nv, __fsqrt_rn(vv));
  return __fadd_rn(ao, __fmul_rn(clamp01(__fsub_rn(ndotv, p.bias)), clamp01(fall)));
}

// The AO of lane `src`'s pixel as the specification has it, by the whole warp:
// for pixels whose steps or image are too large for the 32-bit texel
// arithmetic of hbao_ao_kernel, and for those whose estimate does not decide
// the result.  Lane i takes sample i (direction i / 4, step i % 4); the sum is
// in that order.
template <bool CacheAware>
__device__ __forceinline__ float ao_by_warp(const HbaoScene& s, const float* __restrict__ depth, const HbaoParams& p,
                                            const AoPixel& mine, const float ray[4], const float2 (*rot)[8], int src) {
  const auto get = [&](float v) { return __shfl_sync(0xffffffffu, v, src); };
  const int lane = threadIdx.x & 31, k = lane & 3;
  const float3 P = f3(get(mine.P.x), get(mine.P.y), get(mine.P.z)), N = f3(get(mine.N.x), get(mine.N.y), get(mine.N.z));
  const float u = get(mine.u), v = get(mine.v), r0 = get(ray[0]), r1 = get(ray[1]), r2 = get(ray[2]), r3 = get(ray[3]);
  const int x = __shfl_sync(0xffffffffu, mine.x, src), y = __shfl_sync(0xffffffffu, mine.y, src);
  const float r = k == 0 ? r0 : (k == 1 ? r1 : (k == 2 ? r2 : r3));
  const float2 d = rot[(y & 3) * 4 + (x & 3)][lane >> 2];
  const float kx = rintf(__fmul_rn(r, d.x)), ky = rintf(__fmul_rn(r, d.y));
  const float su = __fadd_rn(__fmul_rn(kx, mine.su_scale), u), sv = __fadd_rn(__fmul_rn(ky, mine.sv_scale), v);
  // Offsets beyond the image only select the clamped edge texel.
  const int ix = int(fminf(fmaxf(kx, -65536.0f), 65536.0f)), iy = int(fminf(fmaxf(ky, -65536.0f), 65536.0f));
  const float zs = CacheAware ? layer_depth(s, depth, (x >> 2) + ix, (y >> 2) + iy, x & 3, y & 3)
                              : depth_at(s, depth, x + ix, y + iy);
  const float3 V = sub(view_pos(s, su, sv, zs), P);
  const float vv = dot3(V, V);
  const float c = ao_add(p, 0.0f, vv, dot3(N, V), __fadd_rn(__fmul_rn(vv, p.neg_inv_r2), 1.0f));
  float ao = 0.0f;
  for (uint32_t m = __ballot_sync(0xffffffffu, c != 0.0f); m; m &= m - 1u)
    ao = __fadd_rn(ao, __shfl_sync(0xffffffffu, c, __ffs(int(m)) - 1));
  return ao;
}

// AO per pixel.  Classic: the pixel's own view position and reconstructed
// normal, samples at full resolution, the 16-bit jitter of texel
// (x & 3, y & 3).  CacheAware: the pixel belongs to deinterleaved layer
// (x & 3, y & 3) at quarter-resolution texel (x >> 2, y >> 2); its uv is that
// texel's centre in the layer, its normal the reconstructed one through an
// RGBA8 store, its samples are texels of the same layer at quarter-resolution
// steps (radius / 4), its jitter the layer's unquantized one; the result
// lands at the pixel, which is the reinterleave.  Special: (AO, view depth)
// stored as two halves.
//
// Bound by instruction issue: 32 samples per pixel, their depths served by L1
// (a 16 x 16 tile's samples overlap).  Per sample, what the arithmetic fixes
// is about 45 operations; the rest was cut: the rotated directions come from a
// table, the four ray lengths are shared by the eight directions, a sample's
// offset is rounded to an integer by adding 1.5 * 2^23 (which leaves the
// integer in the low bits: no conversion instructions, a quarter of the rate
// here), texels are addressed in 32 bits, and two samples of a direction go
// through the float arithmetic as register pairs.  Where the result is a byte,
// a sample's N.V / |V| is first taken with the approximate reciprocal root (2
// instructions for about 30), the error of the sum is bounded, and the few
// pixels whose byte the bound leaves open (one in 500) are done again in full, a
// warp to a pixel; with halves (Special) it would leave one in 50 open, so every
// sample is done in full.
template <bool CacheAware, bool Special>
__global__ void __launch_bounds__(256, 5)
    hbao_ao_kernel(const HbaoScene* __restrict__ scenes, const __grid_constant__ HbaoScene one, int count,
                   const float* __restrict__ depth, uint32_t* color, void* q, const __grid_constant__ HbaoParams p) {
  __shared__ float2 s_rot[16][8];  // rotated directions of jitter texel j
  if (threadIdx.x < 128) {
    const int t = threadIdx.x >> 3, d = threadIdx.x & 7;
    const float* j = (CacheAware ? p.jitter_f : p.jitter) + 4 * t;
    const float dc = p.dirs[2 * d], ds = p.dirs[2 * d + 1];
    s_rot[t][d] = make_float2(__fsub_rn(__fmul_rn(dc, j[0]), __fmul_rn(ds, j[1])),
                              __fadd_rn(__fmul_rn(dc, j[1]), __fmul_rn(ds, j[0])));
  }
  int local = blockIdx.x;
  const HbaoScene* scene = &one;
  if (scenes)
    scene = scenes + scene_of_block<&HbaoScene::block0>(scenes, count, &local);
  else
    __syncthreads();
  const HbaoScene s = *scene;
  const int tiles_x = (s.w + kAoTile - 1) / kAoTile;
  int x = (local % tiles_x) * kAoTile + (int(threadIdx.x) & (kAoTile - 1));
  int y = (local / tiles_x) * kAoTile + int(threadIdx.x) / kAoTile;
  // Lanes beside the image stay for the warp's sake, at an edge pixel; a warp of them
  // leaves (256 views of 33 x 33, cache-aware: 76 us with them, 68 without).
  const bool valid = x < s.w && y < s.h;
  if (!__any_sync(0xffffffffu, valid)) return;
  x = min(x, s.w - 1);
  y = min(y, s.h - 1);
  AoPixel a;
  a.x = x;
  a.y = y;
  a.u = __fdiv_rn(__fadd_rn(float(x), 0.5f), float(s.w));
  a.v = __fdiv_rn(__fadd_rn(float(y), 0.5f), float(s.h));
  a.P = view_pos(s, a.u, a.v, depth_at(s, depth, x, y));
  float inv_len;
  const float3 c = reconstruct_normal(s, depth, x, y, a.u, a.v, s.inv_w, s.inv_h, a.P, inv_len);
  float radius;
  a.su_scale = s.inv_w;
  a.sv_scale = s.inv_h;
  const int ox = x & 3, oy = y & 3, qx = x >> 2, qy = y >> 2, jt = oy * 4 + ox;
  if (!CacheAware) {
    a.N = f3(-__fmul_rn(c.x, inv_len), -__fmul_rn(c.y, inv_len), -__fmul_rn(c.z, inv_len));
    radius = __fdiv_rn(s.radius_to_screen, s.ortho ? 1.0f : a.P.z);
  } else {
    const float e[3] = {c.x, c.y, c.z};
    float n[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      const uint32_t enc = unorm8(__fadd_rn(__fmul_rn(__fmul_rn(e[k], inv_len), 0.5f), 0.5f));
      n[k] = -__fsub_rn(__fmul_rn(byte_unit(enc), 2.0f), 1.0f);
    }
    a.N = f3(n[0], n[1], n[2]);
    a.u = __fmul_rn(__fadd_rn(__fmul_rn(float(qx), 4.0f), __fadd_rn(float(ox), 0.5f)), __fdiv_rn(s.inv_qw, 4.0f));
    a.v = __fmul_rn(__fadd_rn(__fmul_rn(float(qy), 4.0f), __fadd_rn(float(oy), 0.5f)), __fdiv_rn(s.inv_qh, 4.0f));
    a.P = view_pos(s, a.u, a.v, a.P.z);
    radius = __fdiv_rn(__fdiv_rn(s.radius_to_screen, s.ortho ? 1.0f : a.P.z), 4.0f);
    a.su_scale = s.inv_qw;
    a.sv_scale = s.inv_qh;
  }
  const float step = __fdiv_rn(radius, 5.0f);
  float ray[4];
  ray[0] = __fadd_rn(__fmul_rn((CacheAware ? p.jitter_f : p.jitter)[4 * jt + 2], step), 1.0f);
#pragma unroll
  for (int k = 1; k < 4; ++k) ray[k] = __fadd_rn(ray[k - 1], step);
  float ao = 0.0f;
  // Directions have components of at most 1 (and a rounding): offsets stay
  // below 2^22, where adding 1.5 * 2^23 rounds to the nearest integer, ties
  // to even, as rintf does.
  const bool near = s.fits && fabsf(ray[0]) < 2097152.0f && fabsf(ray[3]) < 2097152.0f;
  const bool estimated = near && !Special;
  if (near) {
    const float* img = depth + s.offset;
    const int pitch = int(s.pitch);
    constexpr float kRound = 12582912.0f;
    constexpr int kRoundBits = 0x4B400000;
    const int bx = (CacheAware ? qx : x) - kRoundBits, by = (CacheAware ? qy : y) - kRoundBits;
    const int mx = (CacheAware ? s.qw : s.w) - 1, my = (CacheAware ? s.qh : s.h) - 1;
    const F2 round = f2(kRound), unround = f2(-kRound), su_scale = f2(a.su_scale), sv_scale = f2(a.sv_scale),
             u2 = f2(a.u), v2 = f2(a.v), pi0 = f2(s.pi[0]), pi1 = f2(s.pi[1]), pi2 = f2(s.pi[2]), pi3 = f2(s.pi[3]),
             px = f2(-a.P.x), py = f2(-a.P.y), pz = f2(-a.P.z), nx = f2(a.N.x), ny = f2(a.N.y), nz = f2(a.N.z),
             falloff = f2(p.neg_inv_r2), unit = f2(1.0f);
    const F2 rays[2] = {f2(ray[0], ray[1]), f2(ray[2], ray[3])};
    const auto texel = [&](float tx, float ty) {
      const int ix = min(max(bx + __float_as_int(tx), 0), mx), iy = min(max(by + __float_as_int(ty), 0), my);
      float z;
      if (CacheAware) {
        const int fx = 4 * ix + ox, fy = 4 * iy + oy;
        z = fx < s.w && fy < s.h ? __ldg(img + (fy * pitch + fx)) : 0.0f;
      } else {
        z = __ldg(img + (iy * pitch + ix));
      }
      return z == 0.0f ? s.far_plane : z;
    };
#pragma unroll 2
    for (int d = 0; d < 8; ++d) {
      const float2 rot = s_rot[jt][d];
      const F2 rx = f2(rot.x), ry = f2(rot.y);
#pragma unroll
      for (int k = 0; k < 2; ++k) {
        const F2 tx = add2(mul2(rays[k], rx), round), ty = add2(mul2(rays[k], ry), round);
        const float2 sx = split(tx), sy = split(ty);
        const F2 z = f2(texel(sx.x, sy.x), texel(sx.y, sy.y));
        const F2 zk = s.ortho ? unit : z;
        const F2 su = add2(mul2(add2(tx, unround), su_scale), u2), sv = add2(mul2(add2(ty, unround), sv_scale), v2);
        const F2 Vx = add2(mul2(add2(mul2(su, pi0), pi2), zk), px), Vy = add2(mul2(add2(mul2(sv, pi1), pi3), zk), py),
                 Vz = add2(z, pz);
        if (Special) {
          const F2 vv = add2(add2(mul2(Vx, Vx), mul2(Vy, Vy)), mul2(Vz, Vz));
          const F2 nv = add2(add2(mul2(nx, Vx), mul2(ny, Vy)), mul2(nz, Vz));
          const float2 l = split(vv), n = split(nv), f = split(add2(mul2(vv, falloff), unit));
          ao = ao_add(p, ao, l.x, n.x, f.x);
          ao = ao_add(p, ao, l.y, n.y, f.y);
        } else {
          const float2 l = split(fma2(Vz, Vz, fma2(Vy, Vy, mul2(Vx, Vx))));
          const F2 nv = fma2(nz, Vz, fma2(ny, Vy, mul2(nx, Vx)));
          const float2 n = split(mul2(nv, f2(rsqrt_approx(l.x), rsqrt_approx(l.y))));
          ao = __fmaf_rn(__saturatef(n.x - p.bias), __saturatef(__fmaf_rn(l.x, p.neg_inv_r2, 1.0f)), ao);
          ao = __fmaf_rn(__saturatef(n.y - p.bias), __saturatef(__fmaf_rn(l.y, p.neg_inv_r2, 1.0f)), ao);
        }
      }
    }
  }
  // A byte result (or three, without the blur) is decided by the occlusion at
  // both ends of the estimate's error unless they round differently: the sum's
  // (kAoSumError), 4e-7 for the two roundings of either side that make it an
  // occlusion and the one of each end, and poly_pow's own (kAoPowSlack).
  const long long at = s.offset + (long long)y * s.pitch + x;
  const bool byte_plane = !Special && (!p.no_blur || CacheAware);  // the result is a byte first
  bool open = !near;
  uint32_t result = 0;
  if (estimated) {
    const float est = 1.0f - 2.0f * p.ao_scale * ao;
    const float err = 2.0f * p.ao_scale * (kAoSumError + kAoSumRelative * ao) + 4e-7f;
    const float slack = kAoPowSlack + kAoPowSlackPerExponent * p.pow_exp;
    const float lo = poly_pow(clamp01(est - err), p.pow_exp) - slack, hi = poly_pow(clamp01(est + err), p.pow_exp) + slack;
    if (byte_plane) {
      result = unorm8(lo);
      open = result != unorm8(hi);
    } else {
      const uint32_t old = color[at];
      result = modulate(old, lo);
      open = result != modulate(old, hi);
    }
  }
  for (uint32_t m = __ballot_sync(0xffffffffu, open && valid); m; m &= m - 1u) {
    const int src = __ffs(int(m)) - 1;
    const float v = ao_by_warp<CacheAware>(s, depth, p, a, ray, s_rot, src);
    if ((int(threadIdx.x) & 31) == src) ao = v;
  }
  if (!valid) return;
  if (open || !estimated) {
    const float occl = poly_pow(clamp01(__fsub_rn(1.0f, __fmul_rn(__fmul_rn(ao, p.ao_scale), 2.0f))), p.pow_exp);
    if (Special)
      result = pack_half2(occl, a.P.z);
    else
      result = byte_plane ? unorm8(occl) : modulate(color[at], occl);
  }
  if (p.no_blur)  // the cache-aware result reaches the colour through its 8-bit layers
    color[at] = CacheAware ? modulate(color[at], byte_unit(result)) : result;
  else if (Special)
    static_cast<uint32_t*>(q)[at] = result;
  else
    static_cast<uint8_t*>(q)[at] = uint8_t(result);
}

constexpr int kBlurThreads = 512;

// Weight of the pair of taps r pixels apart whose depths differ by d.
__device__ __forceinline__ float blur_weight(int r, float d, float sharpness) {
  constexpr float falloff = 1.0f / (2.0f * 1.5f * 1.5f);
  const float dd = __fmul_rn(d, sharpness);
  const float rf = float(r);
  return poly_exp2(__fsub_rn(__fmul_rn(__fmul_rn(-rf, rf), falloff), __fmul_rn(dd, dd)));
}

// Both weights at once: taps ra and rb pixels apart, depths differing by a and b.
__device__ __forceinline__ float2 blur_weights(int ra, int rb, float a, float b, float sharpness) {
  constexpr float falloff = 1.0f / (2.0f * 1.5f * 1.5f);
  const F2 d = f2(a, b), up = mul2(d, f2(sharpness)), down = mul2(d, f2(-sharpness));
  const float fa = float(ra), fb = float(rb);
  return poly_exp2(add2(f2(__fmul_rn(__fmul_rn(-fa, fa), falloff), __fmul_rn(__fmul_rn(-fb, fb), falloff)),
                        mul2(up, down)));
}

// Both 7-tap passes, x then y, and the colour multiply.  Bilateral: 8-bit AO
// between the passes, the depths from the linear-depth plane.  Special: (AO,
// depth) halves throughout.
//
// Bound by instruction issue, the exponentials of the tap weights first.  A
// weight depends on the pair of taps alone (the depth difference enters
// squared), so each is computed once for both: along x a lane makes the three
// to its right and takes those to its left from the lanes there (the tile's
// left halo from a small table); along y the weights of a row with the three
// rows above it go through shared memory: 7.3 exponentials per pixel, the
// tile's halo included, instead of 12, two at a time.  One 32 x 32 tile per block with 3
// pixels of halo, clamped at the image's edges as the taps are, so that the
// first pass's result stays in shared memory; 512 threads, because one image
// is a few hundred tiles and the rows of a tile are what hides latency.
template <bool Special>
__global__ void __launch_bounds__(kBlurThreads, 4)
    hbao_blur_kernel(const HbaoScene* __restrict__ scenes, const __grid_constant__ HbaoScene one, int count,
                     const float* __restrict__ depth, const void* __restrict__ q, uint32_t* color,
                     const __grid_constant__ HbaoParams p) {
  constexpr int R = 3, kSide = kBlurTile + 2 * R, kWarps = kBlurThreads / 32;
  __shared__ float s_d[kSide][kSide + 1], s_a[kSide][kSide + 1], s_q[kSide][kBlurTile + 1], s_left[kSide][6];
  __shared__ float s_w[R][kSide][kBlurTile];  // weight of rows (t, t + r): s_w[r - 1][t]
  int local = blockIdx.x;
  const HbaoScene* scene = &one;
  if (scenes) scene = scenes + scene_of_block<&HbaoScene::blur0>(scenes, count, &local);
  const HbaoScene s = *scene;
  const int tiles_x = (s.w + kBlurTile - 1) / kBlurTile;
  const int x0 = (local % tiles_x) * kBlurTile, y0 = (local / tiles_x) * kBlurTile;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int cols = min(kBlurTile, s.w - x0) + 2 * R, rows = min(kBlurTile, s.h - y0) + 2 * R;
  for (int r = warp; r < rows; r += kWarps) {
    const long long row = s.offset + (long long)min(max(y0 + r - R, 0), s.h - 1) * s.pitch;
    for (int c = lane; c < cols; c += 32) {
      const long long at = row + min(max(x0 + c - R, 0), s.w - 1);
      if (Special) {
        const uint32_t v = __ldg(static_cast<const uint32_t*>(q) + at);
        s_a[r][c] = half_lo(v);
        s_d[r][c] = half_hi(v);
      } else {
        const float z = __ldg(depth + at);
        s_a[r][c] = byte_unit(__ldg(static_cast<const uint8_t*>(q) + at));
        s_d[r][c] = z == 0.0f ? s.far_plane : z;
      }
    }
  }
  __syncthreads();
  // Weights between the left halo and the tile: pairs (c, c + r), c < 3 <= c + r.
  for (int i = threadIdx.x; i < rows * 6; i += kBlurThreads) {
    const int row = i / 6, k = i % 6;  // k: r = 1 | r = 2, c = 1, 2 | r = 3, c = 0, 1, 2
    const int r = k == 0 ? 1 : (k < 3 ? 2 : 3), c = k == 0 ? 2 : (k < 3 ? k : k - 3);
    s_left[row][k] = blur_weight(r, __fsub_rn(s_d[row][c + r], s_d[row][c]), p.sharpness);
  }
  __syncthreads();
  for (int row = warp; row < rows; row += kWarps) {
    const int c = lane + R;
    const float cd = s_d[row][c];
    // Below the tile's last row the depth is that row's: its weights go unused.
    const float* down = &s_d[0][c];
    const float d1 = down[min(row + 1, rows - 1) * (kSide + 1)], d2 = down[min(row + 2, rows - 1) * (kSide + 1)],
                d3 = down[min(row + 3, rows - 1) * (kSide + 1)];
    const float2 w12 = blur_weights(1, 2, __fsub_rn(s_d[row][c + 1], cd), __fsub_rn(s_d[row][c + 2], cd), p.sharpness),
                 w3d = blur_weights(3, 1, __fsub_rn(s_d[row][c + 3], cd), __fsub_rn(d1, cd), p.sharpness),
                 d23 = blur_weights(2, 3, __fsub_rn(d2, cd), __fsub_rn(d3, cd), p.sharpness);
    s_w[0][row][lane] = w3d.y;
    s_w[1][row][lane] = d23.x;
    s_w[2][row][lane] = d23.y;
    const float w[3] = {w12.x, w12.y, w3d.x};
    float ct = s_a[row][c], wt = 1.0f;
#pragma unroll
    for (int r = 1; r <= 3; ++r) {
      wt = __fadd_rn(wt, w[r - 1]);
      ct = __fadd_rn(ct, __fmul_rn(s_a[row][c + r], w[r - 1]));
    }
#pragma unroll
    for (int r = 1; r <= 3; ++r) {
      const int base = r == 1 ? 0 : (r == 2 ? 1 : 3);
      float wl = __shfl_up_sync(0xffffffffu, w[r - 1], r);
      if (lane < r) wl = s_left[row][base + lane];
      wt = __fadd_rn(wt, wl);
      ct = __fadd_rn(ct, __fmul_rn(s_a[row][c - r], wl));
    }
    const float out = __fdiv_rn(ct, wt);
    s_q[row][lane] = Special ? __half2float(__float2half_rn(out)) : byte_unit(unorm8(out));
  }
  __syncthreads();
  const int x = x0 + lane;
  if (x >= s.w) return;
  for (int row = warp + R; row < rows - R; row += kWarps) {
    float ct = s_q[row][lane], wt = 1.0f;
#pragma unroll
    for (int r = 1; r <= 3; ++r) {
      const float w = s_w[r - 1][row][lane];
      wt = __fadd_rn(wt, w);
      ct = __fadd_rn(ct, __fmul_rn(s_q[row + r][lane], w));
    }
#pragma unroll
    for (int r = 1; r <= 3; ++r) {
      const float w = s_w[r - 1][row - r][lane];
      wt = __fadd_rn(wt, w);
      ct = __fadd_rn(ct, __fmul_rn(s_q[row - r][lane], w));
    }
    const long long at = s.offset + (long long)(y0 + row - R) * s.pitch + x;
    color[at] = modulate(color[at], __fdiv_rn(ct, wt));
  }
}

template <bool CacheAware, bool Special>
void hbao_launch_t(const HbaoScene* d_scenes, const HbaoScene& one, int count, int ao_blocks, int blur_blocks,
                   const float* depth, uint32_t* color, void* q, const HbaoParams& p, cudaStream_t stream) {
  hbao_ao_kernel<CacheAware, Special><<<ao_blocks, 256, 0, stream>>>(d_scenes, one, count, depth, color, q, p);
  if (!p.no_blur)
    hbao_blur_kernel<Special><<<blur_blocks, kBlurThreads, 0, stream>>>(d_scenes, one, count, depth, q, color, p);
}

}  // namespace

// The jitter table before its 16-bit storage: the values the cache-aware
// algorithm passes per layer as a uniform (Hbao.cpp:603-617, 1000).
void hbao_jitter_unquantized(float out[64]) {
  std::mt19937 rmt;  // default seed, as the reference
  for (int i = 0; i < 16; ++i) {
    const float r1 = float(rmt()) / 4294967296.0f;
    const float r2 = float(rmt()) / 4294967296.0f;
    const float angle = 6.28318530718f * r1 / 8.0f;
    out[4 * i + 0] = float(std::cos(double(angle)));
    out[4 * i + 1] = float(std::sin(double(angle)));
    out[4 * i + 2] = r2;
    out[4 * i + 3] = 0.0f;
  }
}

bool hbao_params(const gbr_hbao_config& c, HbaoParams& p, std::string& err) {
  if (c.special_blur && c.no_blur) {
    err = "Hbao: no_blur and special_blur exclude each other (HbaoConfiguration::setNoBlur / setUseSpecialBlur)";
    return false;
  }
  if (c.algorithm != GBR_HBAO_CLASSIC && c.algorithm != GBR_HBAO_CACHE_AWARE) {
    err = "Hbao: unknown algorithm";
    return false;
  }
  if (!std::isfinite(c.radius) || !(c.radius > 0.0f) || !std::isfinite(c.intensity) ||
      !std::isfinite(c.bias) || !(c.bias < 1.0f) || !std::isfinite(c.blur_sharpness)) {
    err = "Hbao: bad configuration";
    return false;
  }
  std::memset(&p, 0, sizeof p);
  const float r = c.radius;  // metres to view space: 1
  const float r2 = r * r;
  p.neg_inv_r2 = -1.0f / r2;
  p.pow_exp = std::max(c.intensity, 0.0f);
  p.bias = std::min(std::max(c.bias, 0.0f), 1.0f);
  p.bias2 = p.bias >= 1e-4f ? p.bias * p.bias * (1.0f - 1e-5f) : 0.0f;
  p.ao_scale = 1.0f / (1.0f - p.bias) / 32.0f;
  p.sharpness = c.blur_sharpness / 1.0f;
  p.no_blur = c.no_blur ? 1 : 0;
  p.special = c.special_blur ? 1 : 0;
  p.cache_aware = c.algorithm == GBR_HBAO_CACHE_AWARE ? 1 : 0;
  gbr_hbao_jitter_table(p.jitter);
  hbao_jitter_unquantized(p.jitter_f);
  for (int d = 0; d < 8; ++d) {
    const float a = 2.0f * 3.14159265f / 8.0f * float(d);
    p.dirs[2 * d] = float(std::cos(double(a)));
    p.dirs[2 * d + 1] = float(std::sin(double(a)));
  }
  return true;
}

HbaoScene hbao_scene(const float* m, int w, int h, long long offset, long long pitch, float radius) {
  HbaoScene s{};
  s.offset = offset;
  s.pitch = pitch;
  s.w = w;
  s.h = h;
  s.qw = (w + 3) / 4;
  s.qh = (h + 3) / 4;
  s.inv_w = 1.0f / float(w);
  s.inv_h = 1.0f / float(h);
  s.fits = w <= 65536 && h <= 65536 && (long long)h * pitch < (1LL << 31);
  s.inv_qw = 1.0f / float(s.qw);
  s.inv_qh = 1.0f / float(s.qh);
  const float p00 = m[0], p11 = m[5], p20 = m[8], p21 = m[9], p22 = m[10], p30 = m[12], p31 = m[13],
              p32 = m[14];
  s.ortho = m[15] != 0.0f ? 1 : 0;
  s.pi[0] = 2.0f / p00;
  s.pi[1] = 2.0f / p11;
  if (s.ortho) {
    s.pi[2] = -(1.0f + p30) / p00;
    s.pi[3] = -(1.0f - p31) / p11;
    s.far_plane = (p32 - 1.0f) / p22;
    s.radius_to_screen = radius * 0.5f * (float(h) / s.pi[1]);
  } else {
    s.pi[2] = -(1.0f - p20) / p00;
    s.pi[3] = -(1.0f + p21) / p11;
    s.far_plane = p32 / (p22 + 1.0f);
    s.radius_to_screen = radius * 0.5f * (0.5f * float(h) * p00);
  }
  return s;
}

cudaError_t hbao_launch(const HbaoScene* d_scenes, const HbaoScene& one, int count, int ao_blocks,
                        int blur_blocks, const float* depth, uint32_t* color, void* q, const HbaoParams& p,
                        cudaStream_t stream) {
  if (count <= 0 || ao_blocks <= 0) return cudaSuccess;
  const auto launch = p.cache_aware ? (p.special ? hbao_launch_t<true, true> : hbao_launch_t<true, false>)
                                    : (p.special ? hbao_launch_t<false, true> : hbao_launch_t<false, false>);
  launch(d_scenes, one, count, ao_blocks, blur_blocks, depth, color, q, p, stream);
  return cudaGetLastError();
}

}  // namespace gbr

extern "C" {

void gbr_hbao_config_init(gbr_hbao_config* c) {
  if (!c) return;
  std::memset(c, 0, sizeof(*c));
  c->intensity = 0.732f;
  c->bias = 0.05f;
  c->radius = 1.84f;
  c->blur_sharpness = 10.0f;
}

gbr_status gbr_hbao_jitter_table(float out[64]) {
  if (!out) {
    gbr::set_last_error("null argument: out");
    return GBR_ERROR_INVALID_ARGUMENT;
  }
  std::mt19937 rmt;  // default seed, as the reference
  for (int i = 0; i < 16; ++i) {
    const float r1 = float(rmt()) / 4294967296.0f;
    const float r2 = float(rmt()) / 4294967296.0f;
    const float angle = 6.28318530718f * r1 / 8.0f;
    // cos / sin evaluated in double and rounded (the reference uses the
    // float functions; the 16-bit storage below hides the difference).
    const float v[3] = {float(std::cos(double(angle))), float(std::sin(double(angle))), r2};
    // RGBA16 snorm storage: round(v * 32767) / 32767, halves away from zero.
    for (int k = 0; k < 3; ++k) out[4 * i + k] = float(std::round(v[k] * 32767.0f)) / 32767.0f;
    out[4 * i + 3] = 0.0f;
  }
  return GBR_OK;
}

gbr_status gbr_hbao_apply(const gbr_hbao_config* config, const float projection[16], const float* depth,
                          uint32_t* color, int32_t w, int32_t h, int64_t pitch, void* stream) {
  if (!config || !projection || !depth || !color) {
    gbr::set_last_error("null argument");
    return GBR_ERROR_INVALID_ARGUMENT;
  }
  if (w <= 0 || h <= 0 || pitch < w || int64_t(w) * h > (int64_t(1) << 31) - 1) {
    gbr::set_last_error("Hbao: bad image size");
    return GBR_ERROR_INVALID_ARGUMENT;
  }
  gbr::HbaoParams p;
  std::string err;
  if (!gbr::hbao_params(*config, p, err)) {
    gbr::set_last_error(err);
    return GBR_ERROR_INVALID_ARGUMENT;
  }
  const gbr::HbaoScene s = gbr::hbao_scene(projection, w, h, 0, pitch, config->radius);
  const cudaStream_t st = static_cast<cudaStream_t>(stream);
  uint8_t* q = nullptr;
  const size_t plane = p.no_blur ? 0 : size_t(pitch) * size_t(h) * size_t(gbr::hbao_plane_bytes(p));
  cudaError_t e = plane ? cudaMalloc(&q, plane) : cudaSuccess;
  if (!e)
    e = gbr::hbao_launch(nullptr, s, 1, int(gbr::hbao_blocks(w, h, gbr::kAoTile)),
                         int(gbr::hbao_blocks(w, h, gbr::kBlurTile)), depth, color, q, p, st);
  if (!e) e = cudaStreamSynchronize(st);
  cudaFree(q);
  if (e) {
    gbr::set_last_error(std::string("Hbao: ") + cudaGetErrorString(e));
    return e == cudaErrorMemoryAllocation ? GBR_ERROR_OUT_OF_MEMORY : GBR_ERROR_CUDA;
  }
  return GBR_OK;
}

}  // extern "C"
