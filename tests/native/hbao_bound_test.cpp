// The bound on the AO kernel's estimated sum (hbao.h): at least the roundings
// counted one by one, and never exceeded over random pixels, with the reciprocal
// root off by its whole documented error, on whichever side makes the sum worse.
#include <cmath>
#include <cstdio>
#include <random>

#include "hbao.h"

using namespace gbr;

static float clamp01(float v) { return std::fmin(std::fmax(v, 0.0f), 1.0f); }

int main() {
  int failures = 0;
  const double u = std::ldexp(1.0, -24), n = 1.0 + std::sqrt(3.0) / 255.0, root = std::exp2(-22.9);
  const double spec = (3 * u + 2.5 * u + u) * n + u + 5 * u + u;
  const double estimate = (3 * u + root + 1.5 * u + u) * n + u + 4 * u;
  if (32 * (spec + estimate) > kAoSumError || 63 * u > kAoSumRelative) {
    std::fprintf(stderr, "counted %g, bound %g\n", 32 * (spec + estimate), double(kAoSumError));
    ++failures;
  }
  std::mt19937_64 rng(7);
  std::uniform_real_distribution<double> unit(0.0, 1.0), sym(-1.0, 1.0);
  std::normal_distribution<double> normal;
  double worst = 0.0;
  for (int trial = 0; trial < 200000; ++trial) {
    double N[3] = {normal(rng), normal(rng), normal(rng)};
    const double scale = (trial % 2 ? n : 1.0) / std::sqrt(N[0] * N[0] + N[1] * N[1] + N[2] * N[2]);
    const float nx = float(N[0] * scale), ny = float(N[1] * scale), nz = float(N[2] * scale);
    const float bias = trial % 3 ? float(unit(rng) * 0.2) : 0.0f, r2 = float(std::exp(6.0 * sym(rng))),
                neg_inv_r2 = -1.0f / r2;
    float a = 0.0f, lo = 0.0f, hi = 0.0f;
    for (int k = 0; k < 32; ++k) {
      // Directions near the normal, where N.V / |V| is largest, among others.
      const double spread = trial % 5 ? 2.0 * unit(rng) : 0.05;
      double V[3] = {N[0] * scale + spread * normal(rng), N[1] * scale + spread * normal(rng),
                     N[2] * scale + spread * normal(rng)};
      const double l = std::sqrt(V[0] * V[0] + V[1] * V[1] + V[2] * V[2]), want = std::sqrt(r2) * unit(rng);
      const float x = float(V[0] / l * want), y = float(V[1] / l * want), z = float(V[2] / l * want);
      const float vv = x * x + y * y + z * z, nv = nx * x + ny * y + nz * z;
      const float fall = vv * neg_inv_r2 + 1.0f;
      if (fall > 0.0f && nv > 0.0f) a += clamp01(nv / std::sqrt(vv) - bias) * clamp01(fall);
      const float ev = std::fma(z, z, std::fma(y, y, x * x)), en = std::fma(nz, z, std::fma(ny, y, nx * x));
      const float f = clamp01(std::fma(ev, neg_inv_r2, 1.0f));
      const double rs = 1.0 / std::sqrt(double(ev));
      lo = std::fma(clamp01(en * float(rs * (1.0 - root)) - bias), f, lo);
      hi = std::fma(clamp01(en * float(rs * (1.0 + root)) - bias), f, hi);
    }
    for (const float e : {lo, hi}) {
      const double off = std::fabs(double(e) - double(a)), bound = kAoSumError + double(kAoSumRelative) * e;
      worst = std::fmax(worst, off / bound);
      if (off > bound) ++failures;
    }
  }
  if (failures) return 1;
  std::printf("ok, worst %.3f of the bound\n", worst);
  return 0;
}
