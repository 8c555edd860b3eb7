// Largest errors of fixmath.h against long double evaluation, printed one per line:
//   exp2neg   |2^-e - result| in units of 2^-56, over exponents in [0, 128)
//   gauss     |tap - result| in units of 2^-56, over m = 1 .. 15, sigma in [1, 8], fr in [-1/2, 3/2]
//   mad       exact product - result in units of the result, and its mean
//   roundtrip |v - to(from(v))| in units of 2^-55 of the value's power of two, over values and scales
//   tofloat   relative error of fix_to_f64 in units of 2^-53
#include <math.h>
#include <stdio.h>
#include <stdlib.h>

#include <random>

#include "fixmath.h"

using namespace cg;

int main() {
  std::mt19937_64 rng(11);
  uint64_t tab[kFixExpTab];
  for (int i = 0; i < kFixExpTab; ++i) tab[i] = fix_exp_entry(i);
  const long double one = ldexpl(1.0L, kFixOne);
  long double worst = 0;
  for (int i = 0; i < 2000000; ++i) {
    uint64_t e = rng() >> (i % 3 == 0 ? 0 : 5);
    if (i < 4 * kFixExpTab) {  // table edges
      e = ((uint64_t)(i / 2) << (kFixExpFrac - kFixExpBits)) - (uint64_t)(i & 1);
      if (i == 1) e = 0;
    }
    const long double x = exp2l(-ldexpl((long double)e, -kFixExpFrac)) * one;
    const long double d = fabsl(x - (long double)fix_exp2neg<kFixOne>(e, tab));
    if (d > worst) worst = d;
  }
  printf("exp2neg %.4Lf\n", worst);

  worst = 0;
  std::uniform_real_distribution<double> U(0.0, 1.0);
  for (int i = 0; i < 400000; ++i) {
    const int m = 1 + i % 15;
    const double sigma = 1.0 + 7.0 * U(rng);
    const double b = (2.0 * sigma) / (2.0 * sigma - 1.0) * ((double)m / M_PI);
    const long double c = 1.0L / (logl(2.0L) * (long double)b);
    const uint64_t c60 = (uint64_t)llrintl(ldexpl(c, 60));
    const int64_t c57 = (int64_t)llrintl(ldexpl(c, 57));
    const double fr = i % 50 == 0 ? (i % 100 ? -0.5 : 1.5) : -0.5 + 2.0 * U(rng);
    const FixGauss g = fix_gauss((int64_t)llrint(ldexp(fr, 61)), c60);
    for (int l = 0; l < 2 * m + 2; ++l) {
      const long double y = (long double)fr + (long double)(m - l);
      const long double d = fabsl(expl(-y * y / (long double)b) * one - (long double)fix_gauss_tap<kFixOne>(g, m - l, (int64_t)(m - l) * (m - l) * c57, tab));
      if (d > worst) worst = d;
    }
  }
  printf("gauss %.4Lf\n", worst);

  long double lo = 0, hi = 0, sum = 0;
  for (int i = 0; i < 1000000; ++i) {
    const int64_t v = (int64_t)rng() >> (5 + i % 20), w = (int64_t)(rng() >> 8) % ((int64_t)1 << kFixOne);
    const __int128 p = (__int128)v * w;
    const long double d = (long double)(p - ((__int128)fix_mul(fix_split(v), fix_split_w(w)) << kFixOne)) / one;
    sum += d;
    if (d < lo) lo = d;
    if (d > hi) hi = d;
  }
  printf("mad %.4Lf %.4Lf mean %.4Lf\n", lo, hi, sum / 1000000);

  lo = hi = sum = 0;
  for (int i = 0; i < 1000000; ++i) {
    const int64_t v = (int64_t)rng() >> (2 + i % 30), w = (int64_t)(rng() >> 2), c = (int64_t)rng() >> 3;
    const __int128 p = (__int128)v * w;
    const long double d = ldexpl((long double)(p - ((__int128)(fix_mad62(c, fix_split32(v), fix_split32(w)) - c) << 64)), -64);
    sum += d;
    if (d < lo) lo = d;
    if (d > hi) hi = d;
  }
  printf("mad62 %.4Lf %.4Lf mean %.4Lf\n", lo, hi, sum / 1000000);

  double rt = 0, tf = 0;
  for (int i = 0; i < 1000000; ++i) {
    const double v = ldexp(U(rng) - 0.5, (int)(rng() % 1600) - 800);
    int ex;
    frexp(v, &ex);
    const int s = 55 - ex;
    const double back = fix_to_f64(fix_from_f64(fix_bits(v), s), s);
    const double e = fabs(back - v) / ldexp(1.0, ex - 55);
    if (e > rt) rt = e;
    const int64_t n = (int64_t)rng() >> (1 + i % 60);
    if (n) {
      const int k = (int)(rng() % 1000) - 500;
      const double t = fix_to_f64(n, k), x = ldexp((double)n, -k);
      const double r = fabs((t - x) / x) * 9007199254740992.0;
      if (r > tf) tf = r;
    }
  }
  if (fix_to_f64(0, 3) != 0.0 || fix_from_f64(fix_bits(0.0), 50) != 0 || fix_from_f64(fix_bits(-0.0), 50) != 0 ||
      fix_from_f64(fix_bits(1e-300), 55) != 0)
    rt = 1e9;
  printf("roundtrip %.4f\ntofloat %.4f\n", rt, tf);
  return 0;
}
