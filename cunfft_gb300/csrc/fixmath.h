// fixmath.h -- integer arithmetic of the FP64 form's gridding kernels.
//
// GB300 runs about 2 FP64 multiply-adds per clock and SM (measured 1.97) against 29
// 32 x 32 -> 64 bit integer multiply-adds (measured): a 56-bit fixed-point product of three
// of them costs a fifth of an FP64 multiply-add.  So the FP64 form grids in fixed point:
// values relative to the largest one of their tile, tap weights in units of 2^-56, sums in
// 64-bit integers (exact, in any order), converted to and from FP64 by integer operations
// on the bits.
//
// Two products.  Interpolation adds many of them in registers and keeps the two orders
// apart (FixSum).  A number v = v1 2^28 + v0, -2^27 <= v0 < 2^27, is a pair of limbs;
//   v w / 2^56 = v1 w1 + (v1 w0 + v0 w1) / 2^28 + v0 w0 / 2^56,
// and the last term, at most a quarter of a unit of the result, is left out.  It is zero on
// average for every weight, as v0 is centred: with 0 <= v0 < 2^28 all cells of a plane shared
// the offset w0 / 2^29, which the other two dimensions' weights add up while the values they
// weigh cancel (3D, m = 12: relative error 4.8e-14 of an interpolation, 1.2e-14 centred).
// Spreading adds one product at a time to a cell in shared memory (fix_mad62): limbs of 32
// bits, v = v1 2^32 + v0 with -2^31 <= v0 < 2^31, weights in units of 2^-62, so that the
// second order's shift is the choice of its high word:
//   v w / 2^64 = v1 w1 + (v1 w0 + v0 w1) / 2^32 + v0 w0 / 2^64.
//
// Compiled for the device (kernels) and the host (their check on the CPU).
#pragma once

#include <stdint.h>
#include <string.h>

#ifdef __CUDACC__
#define CG_FIX_HD __host__ __device__ __forceinline__
#else
#define CG_FIX_HD inline
#endif

namespace cg {

constexpr int kFixLimb = 28;                    // bits of the low limb
constexpr int kFixOne = 2 * kFixLimb;           // weights are in units of 2^-56

struct FixPair {
  int32_t hi, lo;
};

// limbs of a value, |v| < 2^59 - 2^27, and of a weight
CG_FIX_HD FixPair fix_split(int64_t v) {
  FixPair p;
  p.lo = (int32_t)((uint32_t)v << (32 - kFixLimb)) >> (32 - kFixLimb);
  p.hi = (int32_t)((v - p.lo) >> kFixLimb);
  return p;
}
CG_FIX_HD FixPair fix_split_w(int64_t v) { return fix_split(v); }

// c + a b, written as a carry pair: the interpolation takes 6.7 clocks per complex tap and warp
// with it, 7.5 with mad.wide (measured).
CG_FIX_HD int64_t fix_mad32(int32_t a, int32_t b, int64_t c) {
#ifdef __CUDA_ARCH__
  asm("{\n\t.reg .u32 l, h;\n\tmov.b64 {l, h}, %0;\n\tmad.lo.cc.s32 l, %1, %2, l;\n\t"
      "madc.hi.s32 h, %1, %2, h;\n\tmov.b64 %0, {l, h};\n\t}"
      : "+l"(c)
      : "r"(a), "r"(b));
  return c;
#else
  return c + (int64_t)a * b;
#endif
}

// A sum of products in two accumulators: hi in units of the result, lo in units of 2^-28
// of it and starting at half a unit, so that its shift rounds
struct FixSum {
  int64_t hi = 0, lo = 1 << (kFixLimb - 1);
};
CG_FIX_HD void fix_add(FixSum& a, FixPair v, FixPair w) {
  a.hi = fix_mad32(v.hi, w.hi, a.hi);
  a.lo = fix_mad32(v.hi, w.lo, a.lo);
  a.lo = fix_mad32(v.lo, w.hi, a.lo);
}
CG_FIX_HD int64_t fix_round(FixSum a) { return a.hi + (a.lo >> kFixLimb); }

// v w / 2^56 rounded (within one unit of the exact value, zero on average)
CG_FIX_HD int64_t fix_mul(FixPair v, FixPair w) {
  FixSum a;
  fix_add(a, v, w);
  return fix_round(a);
}

// limbs of 32 bits, the low one centred
CG_FIX_HD FixPair fix_split32(int64_t v) {
  FixPair p;
  p.lo = (int32_t)(uint32_t)v;
  p.hi = (int32_t)((v - p.lo) >> 32);
  return p;
}
// c + v w / 2^64 rounded (within 0.75 units of the exact value, zero on average);
// |v|, |w| <= 2^62.  The second order is kept non-negative by 2^62, so that its high word
// adds without a sign extension.
CG_FIX_HD int64_t fix_mad62(int64_t c, FixPair v, FixPair w) {
  int64_t t = fix_mad32(v.hi, w.lo, ((int64_t)1 << 62) + ((int64_t)1 << 31));
  t = fix_mad32(v.lo, w.hi, t);
  return fix_mad32(v.hi, w.hi, c) + (int64_t)(uint32_t)((uint64_t)t >> 32) - ((int64_t)1 << 30);
}

CG_FIX_HD uint64_t fix_mulhi64(uint64_t a, uint64_t b) {
#ifdef __CUDA_ARCH__
  return __umul64hi(a, b);
#else
  return (uint64_t)(((unsigned __int128)a * b) >> 64);
#endif
}
CG_FIX_HD uint32_t fix_mulhi32(uint32_t a, uint32_t b) { return (uint32_t)(((uint64_t)a * b) >> 32); }

CG_FIX_HD uint64_t fix_bits(double v) {
#ifdef __CUDA_ARCH__
  return (uint64_t)__double_as_longlong(v);
#else
  uint64_t b;
  memcpy(&b, &v, sizeof(b));
  return b;
#endif
}
CG_FIX_HD double fix_from_bits(uint64_t b) {
#ifdef __CUDA_ARCH__
  return __longlong_as_double((long long)b);
#else
  double v;
  memcpy(&v, &b, sizeof(v));
  return v;
#endif
}
CG_FIX_HD int fix_clz64(uint64_t v) {
#ifdef __CUDA_ARCH__
  return __clzll((long long)v);
#else
  return v ? __builtin_clzll(v) : 64;
#endif
}

// Biased exponent of |v| from the high word of its bits (2047: infinity or NaN)
CG_FIX_HD int fix_exp_of_hi(uint32_t hi) { return (int)((hi >> 20) & 0x7FFu); }

// v 2^s rounded towards zero, |v 2^s| < 2^62 (a subnormal v counts as zero, which the
// callers' scales make it)
CG_FIX_HD int64_t fix_from_f64(uint64_t b, int s) {
  const int e = (int)((b >> 52) & 0x7FF);
  const uint64_t mant = ((b & 0xFFFFFFFFFFFFFull) | (1ull << 52)) << 10;  // 63 bits
  const int sh = 1085 - s - e;  // v 2^s = +- mant 2^-sh
  const uint64_t r = e == 0 || sh > 63 ? 0u : mant >> (sh & 63);
  return (int64_t)b < 0 ? -(int64_t)r : (int64_t)r;
}

// v 2^-s as a double (rounded to the nearest, ties away from zero), the result normal or zero
CG_FIX_HD double fix_to_f64(int64_t v, int s) {
  const uint64_t a = (uint64_t)(v < 0 ? -v : v);
  const int lz = fix_clz64(a);
  const uint64_t n = a << (lz & 63);                       // leading one at bit 63
  const uint64_t mant = (n >> 11) + ((n >> 10) & 1u);      // 53 bits, maybe 2^53 after rounding
  const uint64_t e = (uint64_t)(1023 + 63 - lz - s - 1);   // the leading one adds 1 to the exponent
  const uint64_t b = (e << 52) + mant;
  return a == 0 ? 0.0 : fix_from_bits(b | ((uint64_t)v & (1ull << 63)));
}

// 2^(-2^-k), k = 1 .. 8, in units of 2^-63
CG_FIX_HD uint64_t fix_root(int k) {
  switch (k) {
    case 1: return 0x5a827999fcef3242ull;
    case 2: return 0x6ba27e656b4eb57aull;
    case 3: return 0x75606373ee921c97ull;
    case 4: return 0x7a92be8a92436616ull;
    case 5: return 0x7d41d96db915019dull;
    case 6: return 0x7e9f06067a4360baull;
    case 7: return 0x7f4f08ae3dc7c426ull;
    default: return 0x7fa765aca88f6453ull;
  }
}
constexpr int kFixExpBits = 8;
constexpr int kFixExpTab = 1 << kFixExpBits;

// Entry i of the exponential's table: 2^(-i / 256) in units of 2^-62 (at most 8 roundings)
CG_FIX_HD uint64_t fix_exp_entry(int i) {
  uint64_t t = 1ull << 63;
  for (int k = 1; k <= kFixExpBits; ++k)
    if (i & (kFixExpTab >> k)) t = fix_mulhi64(t, fix_root(k)) << 1;
  return (t + 1u) >> 1;
}

constexpr int kFixExpFrac = 57;  // exponents are in units of 2^-57, below 2^7

// 2^-e in units of 2^-BITS (BITS <= 62), e in units of 2^-57: table of 2^(-i/256) times exp(-x),
// x = ln 2 times the remainder (below 2^-8.5), by its Taylor series to x^5, terms past x^2
// in 32-bit arithmetic (table-driven exponential, P. T. P. Tang, ACM TOMS 15, 1989).
// Within 0.2 units of 2^-56 and the last rounding of the exact value.
template <int BITS>
CG_FIX_HD int64_t fix_exp2neg(uint64_t e, const uint64_t* tab) {
  const int ei = (int)(e >> kFixExpFrac);
  const uint64_t T = tab[(e >> (kFixExpFrac - kFixExpBits)) & (kFixExpTab - 1)];
  const uint64_t r = e & ((1ull << (kFixExpFrac - kFixExpBits)) - 1);
  const uint64_t X = fix_mulhi64(r << 15, 0xb17217f7d1cf79acull);  // x 2^72
  const uint64_t Y = fix_mulhi64(X, X);                            // x^2 2^80
  const uint32_t xh = (uint32_t)(X >> 32), xs = (uint32_t)(X >> 40);  // x 2^40, x 2^32
  const uint32_t q = 0x55555555u - fix_mulhi32(xs, 0x15555555u - fix_mulhi32(xs, 0x4444444u));  // 1/3 - x/12 + x^2/60
  const uint32_t z = (uint32_t)(((uint64_t)xh * q) >> 30);         // x q 2^42
  const uint64_t t = (Y >> 1) - (((uint64_t)(uint32_t)(Y >> 31) * z) >> 12);  // x^2/2 (1 - x q), 2^80
  const uint64_t d = (X >> 8) - (t >> 16);                         // 1 - exp(-x), 2^64
  const uint64_t v = T - fix_mulhi64(T, d);                        // units of 2^-62
  const int sh = 62 - BITS + ei;
  return sh > 62 ? 0 : (int64_t)((v + ((1ull << sh) >> 1)) >> sh);
}

// Gaussian taps exp(-(fr + k)^2 / b) = 2^-(P + k Q + k^2 c): per node and dimension
// P = c fr^2 and Q = 2 c fr, c = log2(e) / b, all in units of 2^-57.  fr in (-2, 2) in units
// of 2^-61; c60 = c 2^60 (c < 8).
struct FixGauss {
  int64_t P, Q;
};
CG_FIX_HD FixGauss fix_gauss(int64_t fr61, uint64_t c60) {
  const uint64_t a = (uint64_t)(fr61 < 0 ? -fr61 : fr61);
  const uint64_t f2 = fix_mulhi64(a << 1, a << 1);       // fr^2 2^60
  FixGauss g;
  g.P = (int64_t)(fix_mulhi64(f2 << 2, c60) >> 1);       // (2^62 2^60 / 2^64) / 2
  const int64_t h = (int64_t)(fix_mulhi64(a << 2, c60 << 1) >> 2);  // c fr 2^60 -> 2 c fr 2^59 -> 2^57
  g.Q = fr61 < 0 ? -h : h;
  return g;
}
// k2c = k^2 c in units of 2^-57
template <int BITS>
CG_FIX_HD int64_t fix_gauss_tap(FixGauss g, int k, int64_t k2c, const uint64_t* tab) {
  const uint64_t e = (uint64_t)(g.P + k2c + (int64_t)k * g.Q);
  return fix_exp2neg<BITS>(e > ~0ull - (1ull << 50) ? 0u : e, tab);  // rounding may leave e just below zero
}

}  // namespace cg
