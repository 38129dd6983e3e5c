// Host restatement of the FP64 face quotients (drnum_b200/csrc/fv_f64.cuh):
// the kernel's own code with the device intrinsics as IEEE operations and the
// reciprocal seed as 1/b, off by a chosen error and cut to its upper 32 bits.
// Counts quotients the guard lets pass that differ from `/`; exits 1 if any.
//
// The denominators lie just below 2 (times a power of two), where rounding the
// reciprocal leaves the least room, from inside the guard's excluded set down,
// and their reciprocals next to the midpoint of two doubles; the numerators put
// the quotient next to one.
#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <random>

#define __device__
#define __forceinline__ inline
#define __noinline__
using std::max;
using std::min;
static uint64_t bits(double x) { uint64_t u; std::memcpy(&u, &x, 8); return u; }
static double from_bits(uint64_t u) { double x; std::memcpy(&x, &u, 8); return x; }
static double __fma_rn(double a, double b, double c) { return std::fma(a, b, c); }
static double __dmul_rn(double a, double b) { return a * b; }
static double __dadd_rn(double a, double b) { return a + b; }
static double __dsub_rn(double a, double b) { return a - b; }
static int __double2hiint(double x) { return (int)(bits(x) >> 32); }
static int __double2loint(double x) { return (int)(uint32_t)bits(x); }
static double __hiloint2double(int h, int l) { return from_bits((uint64_t)(uint32_t)h << 32 | (uint32_t)l); }
static float __int_as_float(int i) { float f; std::memcpy(&f, &i, 4); return f; }

namespace dn {
static double seed_error = 0;   // relative
static double rcp_seed(double b) { return from_bits(bits((1.0 + seed_error) / b) & 0xffffffff00000000ull); }
static float max_nan(float a, float b, float c)
{
  return a != a || b != b || c != c ? NAN : max(a, max(b, c));
}
}
#include "fv_f64.cuh"

typedef unsigned __int128 u128;

// k / 2^54 modulo odd b
static uint64_t over_2_54(uint64_t k, uint64_t b)
{
  uint64_t x = k % b;
  for (int n = 0; n < 54; ++n) x = x & 1 ? (x >> 1) + (b >> 1) + 1 : x >> 1;
  return x;
}

static long bad = 0, passed = 0, guarded = 0;

static void check(double a, double b)
{
  dn::Guard g;
  const dn::Recip r(b, g);
  const double q = r.quot(a), i = r.inverse();
  // the limiter's halved quotient d2 / b (b = r r + 1 there, so b itself as the first denominator)
  const double d1[1] = {b}, d2[1] = {a};
  double h[1];
  dn::half_van_albada(d1, d2, h, g);
  if (g.any()) { ++guarded; return; }
  ++passed;
  const double t = a / b;
  if (q != t || i != 1.0 / b || 2.0 * h[0] != (t * t + t) / (t * t + 1.0)) {
    if (bad++ < 5) std::printf("%a / %a with the seed off by %g: %a, %a\n", a, b, dn::seed_error, q, t);
  }
}

// the seed's largest error at these denominators (f64_seed.cu)
static const double kSeed = std::exp2(-20.9);

int main(int argc, char** argv)
{
  const long n = argc > 1 ? std::atol(argv[1]) : 200000;
  for (int k = -64; k <= 64; ++k) {   // one unit off with a seed off by 2^-19.96
    dn::seed_error = k * kSeed / 64;
    check(0x1.19e5f1ca8a7e7p+52, 0x1.ffffee5d645adp+52);
  }
  std::mt19937_64 rng(7);
  std::uniform_real_distribution<double> error(-kSeed, kSeed), range(0, 16);
  for (long m = 0; m < n; ++m) {
    // significand 2^53 - s, s odd: its reciprocal is 2^-53 (2^52 + s/2 + s^2 2^-54)/2^52 and more, next to
    // a midpoint for s^2 next to a multiple j of 2^54; j log-uniform
    const double j = std::floor(std::exp2(range(rng)));
    const uint64_t s = ((uint64_t)std::rint(std::sqrt(j) * 0x1p27) & ~3ull) + (rng() & 3) | 1;
    const uint64_t b = (1ull << 53) - s;
    // of some seeds the one with the worst reciprocal
    double worst = 0, seed = 0;
    for (int v = 0; v < 24; ++v) {
      dn::seed_error = v < 2 ? (v ? kSeed : -kSeed) : error(rng);
      dn::Guard g;
      const double e = std::fabs(std::fma(-(double)b, dn::Recip((double)b, g).y, 1.0));
      if (e > worst) { worst = e; seed = dn::seed_error; }
    }
    dn::seed_error = seed;
    // a 2^54 - b (odd) = +-1, +-3: a/b is that many units of 1/b off a midpoint
    for (uint64_t k : {uint64_t(1), b - 1, uint64_t(3), b - 3}) {
      const uint64_t a = over_2_54(k, b);
      if (a >> 52) check((double)a, (double)b);
    }
  }
  std::printf("%ld passed, %ld guarded, %ld wrong\n", passed, guarded, bad);
  return bad || !passed || !guarded;
}
