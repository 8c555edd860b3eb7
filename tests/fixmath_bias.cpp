// Largest mean of exact product - fix_mul over values, for any one weight, in units of the
// result; and the largest sum before a limb overflows: v = +-(2^59 - 2^27 - 1) split and joined.
#include <math.h>
#include <stdio.h>

#include <random>

#include "fixmath.h"

using namespace cg;

int main() {
  std::mt19937_64 rng(5);
  long double worst = 0;
  for (int i = 0; i < 200; ++i) {
    const int64_t w = (int64_t)(rng() >> 8) >> (i % 8);
    long double sum = 0;
    for (int k = 0; k < 40000; ++k) {
      const int64_t v = (int64_t)rng() >> 6;
      sum += ldexpl((long double)((__int128)v * w - ((__int128)fix_mul(fix_split(v), fix_split_w(w)) << kFixOne)), -kFixOne);
    }
    if (fabsl(sum / 40000) > worst) worst = fabsl(sum / 40000);
  }
  const int64_t top = ((int64_t)1 << 59) - ((int64_t)1 << 27) - 1;
  for (int64_t v : {top, -top, (int64_t)1 << 27, -((int64_t)1 << 27), (int64_t)0}) {
    const FixPair p = fix_split(v);
    if ((int64_t)p.hi * (1 << kFixLimb) + p.lo != v) worst = 1e9;
  }
  printf("%.5Lf\n", worst);
  return 0;
}
