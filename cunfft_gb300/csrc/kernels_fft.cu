// kernels_fft.cu -- the FP64 form's FFT in fixed point (power-of-two grids).
//
// An FP64 FFT is bound by GB300's FP64 pipe (2 multiply-adds per clock and SM): the library's
// 1024^2 transform takes 172 us, of which memory needs about 10.  Here a CTA transforms C
// neighbouring lines of one dimension in shared memory with 64-bit integers (fixmath.h): each
// line's values are scaled by a power of two of its own (neighbouring lines may belong to
// different instances of a batch) so that no sum can overflow, radix-4 passes
// (Stockham order: twiddle, butterfly, store; one radix-2 pass first when log2 L is odd) with
// twiddles in units of 2^-62, whose product divides by four as the butterfly may multiply by
// four, and FP64 again on the way out.  Where the sum of a line's magnitudes rules that growth
// out, its values are shifted up first, so that a line of few large values keeps its bits too.
// A pass's rounding errors stay below 2^-59 of the bound on its values, for dense lines 2^-54
// of the result.  Lines whose values are not finite, or near FP64's
// exponent limits, take the same passes in FP64.
//
// The forward transform is fused with the roll-off and skips the zero padding: a pass reads
// only the rows that hold coefficients and transforms, along dimension t, only lines with
// nonzero entries (3D: 1/4 + 1/2 + 1 of the work of three full passes); the first pass reads
// the coefficients and applies the roll-off factors.  The adjoint transforms the whole grid
// (the grid stays readable).  1D sizes above 4096 go as n = na nb in two passes through a
// second buffer with the twiddles e^{-+2 pi i kb ia / n} between them.
//
// Bound: integer multiply-adds (9 per point and radix-4 pass at 29 per clock and SM) and the
// 64-bit additions beside them.  Measured, forward with roll-off and
// adjoint: 1024^2 51 and 54 us (library and roll-off kernel: 180 and 173), 128^3 68 and 101 us
// (368 and 356), 2^18 29 and 27 us (96 and 92).  A scale and a sum per
// line cost 5 to 10 % of that (1024^2 49 and 52 us, 128^3 63 and 89 with one scale per CTA).
#include <math.h>

#include <vector>

#include "fixmath.h"
#include "runtime.h"

namespace cg {

constexpr int kFftThreads = 256;
constexpr int kFftMaxL = 4096;  // points of a line in shared memory
constexpr int kFftMaxC = 64;    // lines of a CTA, at most (16 points each)

// One pass: FFTs along dimension t of the grid.
struct FftArgs {
  const double2* src;
  double2* dst;
  const int4* tw;       // e^{2 pi i k / L}: cos, sin as limbs of 32 bits in units of 2^-62
  const int4* post_hi;  // 1D, first of two passes: e^{2 pi i k / n} in steps of 2^post_sh ...
  const int4* post_lo;  // ... and within one
  const double* roc;    // roll-off factors (src holds coefficients) or null
  uint32_t lines;
  uint32_t N[kMaxDim];  // sizes of the leading dimensions: coefficients (pad) or grid points
  uint32_t n[kMaxDim];  // their grid sizes
  int64_t lead_n;       // product of n[]
  int64_t valid;        // pad: nonzero entries (coefficients) of a line
  int64_t dst_l;        // second of two 1D passes: destination stride (else 0)
  int pad;              // the zero-padded forward transform
  int nlead;
  int logL, logC, log_tail;  // tail = 2^log_tail lines per leading index: the later dimensions
  int post_sh, post_log;
};

__device__ __forceinline__ FixPair as_pair2(int hi, int lo) {
  FixPair p;
  p.hi = hi;
  p.lo = lo;
  return p;
}

struct I2 {
  int64_t x, y;
};

// v times (c + i s) / 4 (a product of 62-bit limbs); |v| <= 2^61
__device__ __forceinline__ I2 fft_mul(I2 v, int4 w) {
  const FixPair x = fix_split32(v.x), y = fix_split32(v.y), c = as_pair2(w.x, w.y), s = as_pair2(w.z, w.w);
  I2 r;
  int64_t t = fix_mad32(x.hi, c.lo, (int64_t)1 << 31);
  t = fix_mad32(x.lo, c.hi, t);
  t = fix_mad32(y.hi, -s.lo, t);
  t = fix_mad32(y.lo, -s.hi, t);
  r.x = fix_mad32(y.hi, -s.hi, fix_mad32(x.hi, c.hi, t >> 32));
  t = fix_mad32(x.hi, s.lo, (int64_t)1 << 31);
  t = fix_mad32(x.lo, s.hi, t);
  t = fix_mad32(y.hi, c.lo, t);
  t = fix_mad32(y.lo, c.hi, t);
  r.y = fix_mad32(y.hi, c.hi, fix_mad32(x.hi, s.hi, t >> 32));
  return r;
}

// The arithmetic of a pass: integers or FP64.
struct FftFix {
  using V = I2;
  static __device__ __forceinline__ V make(double2 v, int sc) {
    I2 r;
    r.x = fix_from_f64(fix_bits(v.x), sc);
    r.y = fix_from_f64(fix_bits(v.y), sc);
    return r;
  }
  static __device__ __forceinline__ double2 back(V v, int sc) { return make_double2(fix_to_f64(v.x, sc), fix_to_f64(v.y, sc)); }
  static __device__ __forceinline__ V up(V v, int s) {
    I2 r;
    r.x = (int64_t)((uint64_t)v.x << s);
    r.y = (int64_t)((uint64_t)v.y << s);
    return r;
  }
  static __device__ __forceinline__ V mul(V v, int4 w) { return fft_mul(v, w); }
  static __device__ __forceinline__ V quarter(V v) {
    I2 r;
    r.x = (v.x + 2) >> 2;
    r.y = (v.y + 2) >> 2;
    return r;
  }
};
struct FftF64 {
  using V = double2;
  static __device__ __forceinline__ V make(double2 v, int) { return v; }
  static __device__ __forceinline__ double2 back(V v, int) { return v; }
  static __device__ __forceinline__ double2 tw(int4 w) {
    const double u = 2.168404344971009e-19;  // 2^-62
    const double hi = 4294967296.0;
    return make_double2(((double)w.x * hi + (double)w.y) * u, ((double)w.z * hi + (double)w.w) * u);
  }
  static __device__ __forceinline__ V up(V v, int) { return v; }
  static __device__ __forceinline__ V mul(V v, int4 w) {
    const double2 t = tw(w);
    return make_double2(v.x * t.x - v.y * t.y, v.x * t.y + v.y * t.x);
  }
  static __device__ __forceinline__ V quarter(V v) { return v; }
};

template <typename V>
__device__ __forceinline__ V vadd(V a, V b) {
  V r;
  r.x = a.x + b.x;
  r.y = a.y + b.y;
  return r;
}
template <typename V>
__device__ __forceinline__ V vsub(V a, V b) {
  V r;
  r.x = a.x - b.x;
  r.y = a.y - b.y;
  return r;
}

// 4-point DFT of v in place, e^{-+...} (INV: +)
template <bool INV, typename V>
__device__ __forceinline__ void fft4(V* v) {
  const V a = vadd(v[0], v[2]), b = vsub(v[0], v[2]), c = vadd(v[1], v[3]), d = vsub(v[1], v[3]);
  v[0] = vadd(a, c);
  v[2] = vsub(a, c);
  V p, q;  // b - i d, b + i d
  p.x = b.x + d.y;
  p.y = b.y - d.x;
  q.x = b.x - d.y;
  q.y = b.y + d.x;
  v[1] = INV ? q : p;
  v[3] = INV ? p : q;
}

__device__ __forceinline__ int4 fft_tw(const int4* __restrict__ t, int k, bool inv) {
  int4 w = __ldg(t + k);
  if (!inv) {
    w.z = -w.z;
    w.w = -w.w;
  }
  return w;
}

// Room of a line in fixed point: its complex values are below 2^(60.5 - room), and the passes
// to come multiply them by 2^grow at most.
struct FftRoom {
  int room, grow;
  __device__ __forceinline__ void pass(int g) {  // a pass that adds 2^g values
    g = min(g, grow);
    room -= g;
    grow -= g;
  }
};

// The passes over a CTA's lines: v holds, per task u, the points j + r L / 4 of line c.  Returns
// the bits that the divisions took off the scale.
template <typename A, int TPT, bool INV>
__device__ __forceinline__ int fft_passes(typename A::V (&v)[TPT][4], typename A::V* buf, const FftArgs& a, int c, int j0, int dj,
                                          FftRoom& rm) {
  using V = typename A::V;
  const int L4 = 1 << (a.logL - 2), lc = a.logC;
  int ns;
  // first pass: no twiddles
  if (a.logL & 1) {
#pragma unroll
    for (int u = 0; u < TPT; ++u) {
      const int j = j0 + u * dj;
      const V e0 = vadd(v[u][0], v[u][2]), o0 = vsub(v[u][0], v[u][2]);
      const V e1 = vadd(v[u][1], v[u][3]), o1 = vsub(v[u][1], v[u][3]);
      buf[((2 * j) << lc) + c] = e0;
      buf[((2 * j + 1) << lc) + c] = o0;
      buf[((2 * (j + L4)) << lc) + c] = e1;
      buf[((2 * (j + L4) + 1) << lc) + c] = o1;
    }
    ns = 2;
    rm.pass(1);
  } else {
#pragma unroll
    for (int u = 0; u < TPT; ++u) {
      const int j = j0 + u * dj;
      fft4<INV>(v[u]);
#pragma unroll
      for (int r = 0; r < 4; ++r) buf[((4 * j + r) << lc) + c] = v[u][r];
    }
    ns = 4;
    rm.pass(2);
  }
  for (int off = 0;; ns *= 4) {
    __syncthreads();
    const int step = L4 / ns;  // L / (4 ns)
#pragma unroll
    for (int u = 0; u < TPT; ++u) {
      const int j = j0 + u * dj, k = (j & (ns - 1)) * step;
#pragma unroll
      for (int r = 0; r < 4; ++r) {
        const V t = A::up(buf[((j + r * L4) << lc) + c], rm.room);
        v[u][r] = r == 0 ? A::quarter(t) : A::mul(t, fft_tw(a.tw, r * k, INV));
      }
      fft4<INV>(v[u]);
    }
    off += 2 - rm.room;
    rm.room = 2;
    rm.pass(2);
    if (ns == L4) return off;  // the last pass: results at j + r L / 4
    __syncthreads();
#pragma unroll
    for (int u = 0; u < TPT; ++u) {
      const int j = j0 + u * dj, d = ((j & ~(ns - 1)) << 2) + (j & (ns - 1));
#pragma unroll
      for (int r = 0; r < 4; ++r) buf[((d + r * ns) << lc) + c] = v[u][r];
    }
  }
}

template <typename A, int TPT, bool INV>
__device__ __forceinline__ void fft_run(double2 (&in)[TPT][4], unsigned char* smem, const FftArgs& a, int c, int j0, int dj,
                                        int sc, FftRoom rm, bool on, uint32_t tail_i, double2* out, int64_t stride) {
  using V = typename A::V;
  V v[TPT][4];
#pragma unroll
  for (int u = 0; u < TPT; ++u)
#pragma unroll
    for (int r = 0; r < 4; ++r) v[u][r] = A::make(in[u][r], sc);
  const int so = sc - fft_passes<A, TPT, INV>(v, reinterpret_cast<V*>(smem), a, c, j0, dj, rm);  // (FP64: not used)
  const int L4 = 1 << (a.logL - 2);
  if (!on) return;
#pragma unroll
  for (int u = 0; u < TPT; ++u) {
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      const int l = j0 + u * dj + r * L4;
      V t = v[u][r];
      int s = so;
      if (a.post_hi) {
        const int64_t m = ((int64_t)l * tail_i) & (((int64_t)1 << a.post_log) - 1);
        // two divisions by four; the first leaves room for two bits
        t = A::mul(A::up(t, rm.room), fft_tw(a.post_hi, (int)(m >> a.post_sh), INV));
        t = A::mul(A::up(t, 2), fft_tw(a.post_lo, (int)(m & ((1 << a.post_sh) - 1)), INV));
        s -= 2 - rm.room;
      }
      out[l * stride] = A::back(t, s);
    }
  }
}

// |v| rounded up to a multiple of 2^(key - 1040); zero for zero and what the scale makes zero
__device__ __forceinline__ uint32_t fft_mag(double v, int key) {
  const uint32_t hi = (uint32_t)__double2hiint(v), e = fix_exp_of_hi(hi);
  const uint32_t mant = (hi & 0xFFFFFu) | 0x100000u;  // 21 bits
  return e == 0 ? 0u : (mant >> min(31u, 3u + (uint32_t)key - e)) + 1u;
}

template <int TPT, bool INV>
__global__ void __launch_bounds__(kFftThreads, TPT == 4 ? 2 : 3) k_fft(FftArgs a) {
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ uint32_t s_top[kFftMaxC], s_sum[kFftMaxC];  // per line
  __shared__ int s_f64;
  const int C = 1 << a.logC, L = 1 << a.logL, L4 = L >> 2;
  const int c = threadIdx.x & (C - 1), j0 = threadIdx.x >> a.logC, dj = kFftThreads >> a.logC;
  const uint32_t line = blockIdx.x * (uint32_t)C + c;
  const bool on = line < a.lines;
  if (threadIdx.x < C) s_top[threadIdx.x] = s_sum[threadIdx.x] = 0;
  if (threadIdx.x == 0) s_f64 = 0;
  // the line's place: (instance, leading indices) and tail
  const int64_t tail = (int64_t)1 << a.log_tail;
  const uint32_t tail_i = line & (uint32_t)(tail - 1);
  uint32_t rest = line >> a.log_tail, idx[kMaxDim] = {0, 0, 0};
  int64_t lead = 0, mul = 1;
#pragma unroll
  for (int t = kMaxDim - 2; t >= 0; --t) {
    if (t < a.nlead) {
      const uint32_t q = rest / a.N[t], i = rest - q * a.N[t], half = a.N[t] / 2;
      idx[t] = i;
      // coefficient i has frequency i - half, at that index modulo n
      lead += (int64_t)(!a.pad ? i : (i < half ? i + a.n[t] - half : i - half)) * mul;
      mul *= a.n[t];
      rest = q;
    }
  }
  const int64_t base = ((rest * a.lead_n + lead) * L << a.log_tail) + tail_i;
  double fac = 1.0;
  int64_t row = rest, tb = 0;  // roll-off: the line's coefficients and factors
  if (a.roc) {
#pragma unroll
    for (int t = 0; t < kMaxDim - 1; ++t) {
      if (t < a.nlead) {
        fac *= a.roc[tb + idx[t]];
        row = row * a.N[t] + idx[t];
        tb += a.N[t];
      }
    }
  }
  double2 in[TPT][4];
  uint32_t top = 0;
  const int64_t total = (int64_t)L << a.log_tail, half = a.valid / 2;
#pragma unroll
  for (int u = 0; u < TPT; ++u) {
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      const int l = j0 + u * dj + r * L4;
      double2 x = make_double2(0.0, 0.0);
      if (a.roc) {
        const int64_t i = ((int64_t)l << a.log_tail) + tail_i;  // the whole index in 1D
        const int64_t s = i < a.valid - half ? i + half : (i >= total - half ? i - total + half : -1);
        if (on && s >= 0) {
          x = a.src[row * a.valid + s];
          const double f = fac * a.roc[tb + s];
          x.x *= f;
          x.y *= f;
        }
      } else if (on && (!a.pad || l < a.valid - half || l >= L - half)) {
        x = a.src[base + ((int64_t)l << a.log_tail)];
      }
      in[u][r] = x;
      top = max(top, max((uint32_t)__double2hiint(x.x) & 0x7FFFFFFFu, (uint32_t)__double2hiint(x.y) & 0x7FFFFFFFu));
    }
  }
  __syncthreads();
  for (int o = 16; o >= C; o >>= 1) top = max(top, __shfl_xor_sync(0xffffffffu, top, o));  // the warp's lanes of a line
  if ((threadIdx.x & 31) < C) atomicMax(&s_top[c], top);
  __syncthreads();
  top = s_top[c];
  const int key = fix_exp_of_hi(top);
  if (top != 0 && (key < 100 || key > 1900)) s_f64 = 1;
  // sum of the components' magnitudes, rounded up, 2^18 standing for 2^(key - 1022) above the largest
  uint32_t sum = 0;
#pragma unroll
  for (int u = 0; u < TPT; ++u)
#pragma unroll
    for (int r = 0; r < 4; ++r) sum += fft_mag(in[u][r].x, key) + fft_mag(in[u][r].y, key);
  for (int o = 16; o >= C; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
  if ((threadIdx.x & 31) < C) atomicAdd(&s_sum[c], sum);
  __syncthreads();
  sum = s_sum[c];
  const bool f64 = s_f64 != 0;
  double2* out = a.dst + base;
  int64_t stride = tail;
  if (a.dst_l) {  // second 1D pass: line `lead` of instance `rest`, transposed
    out = a.dst + rest * a.lead_n * L + lead;
    stride = a.dst_l;
  }
  // Components below 2^58 (2^59 where the first pass only adds two): with what the first pass
  // adds, complex values stay below 2^60.5.  They never exceed the sum of the line's magnitudes,
  // 2^grow times its largest: what a line of few large values does not grow, its divisions spare.
  FftRoom rm;
  rm.room = 2 - (a.logL & 1);
  rm.grow = sum > (1u << 18) ? 14 - __clz(sum - 1) : 0;
  if (!f64)
    fft_run<FftFix, TPT, INV>(in, smem, a, c, j0, dj, 58 + (a.logL & 1) - (key - 1022), rm, on, tail_i, out, stride);
  else
    fft_run<FftF64, TPT, INV>(in, smem, a, c, j0, dj, 0, rm, on, tail_i, out, stride);
}

// ---------------------------------------------------------------------------
// Host side
// ---------------------------------------------------------------------------
static int ilog2(int64_t v) {
  int l = 0;
  while (((int64_t)1 << l) < v) ++l;
  return l;
}

// cos and sin of 2 pi i / L in units of 2^-62, L a power of two, i <= L / 2
static void root_of_unity(int64_t i, int64_t L, int64_t* c, int64_t* s) {
  if (i * 2 == L) {
    *c = -((int64_t)1 << 62);
    *s = 0;
    return;
  }
  if (i * 4 == L) {
    *c = 0;
    *s = (int64_t)1 << 62;
    return;
  }
  const long double t = 2.0L * acosl(-1.0L) * (long double)i / (long double)L;  // at most pi / 4
  *c = llrintl(ldexpl(cosl(t), 62));
  *s = llrintl(ldexpl(sinl(t), 62));
}

// e^{2 pi i k / L}, k = 0 .. count - 1 (powers of two), appended to the table: entry k is the
// entry without k's top bit times that bit's root, log2 count roundings of 2^-63 at most
static void twiddles(std::vector<int4>& out, int64_t L, int64_t count) {
  std::vector<int64_t> c((size_t)count), s((size_t)count);
  c[0] = (int64_t)1 << 62;
  s[0] = 0;
  const __int128 half = (__int128)1 << 61;
  for (int64_t b = 1; b < count; b *= 2) {
    int64_t rc, rs;
    root_of_unity(b, L, &rc, &rs);
    for (int64_t k = 0; k < b; ++k) {
      c[b + k] = (int64_t)(((__int128)c[k] * rc - (__int128)s[k] * rs + half) >> 62);
      s[b + k] = (int64_t)(((__int128)c[k] * rs + (__int128)s[k] * rc + half) >> 62);
    }
  }
  for (int64_t k = 0; k < count; ++k) {
    FixPair pc = fix_split32(c[k]), ps = fix_split32(s[k]);
    if (pc.lo == INT32_MIN) ++pc.lo;  // the kernels negate limbs
    if (ps.lo == INT32_MIN) ++ps.lo;
    out.push_back(make_int4(pc.hi, pc.lo, ps.hi, ps.lo));
  }
}

void fft_fix_release(Plan& p) {
  cudaFree(p.fx_tab);
  cudaFree(p.fx_tmp);
  p.fx_tab = nullptr;
  p.fx_tmp = nullptr;
  p.fx_on = false;
}

// Tables of the FP64 form's FFT, where it covers the grid: power-of-two sizes of 16 to 4096
// points (1D: to 2^24, with a second buffer of at most 1 GB).  The plan takes the library's
// FFT for everything else, and where the memory cannot be had.
void fft_fix_prepare(Plan& p) {
  const Geom& g = p.geo;
  p.fx_on = false;
  if (p.prec != kF64) return;
  for (int t = 0; t < g.d; ++t)
    if ((g.n[t] & (g.n[t] - 1)) != 0 || g.n[t] < 16 || g.n[t] > (g.d == 1 ? (int64_t)1 << 24 : (int64_t)kFftMaxL)) return;
  const bool two = g.d == 1 && g.n[0] > kFftMaxL;
  if (two && g.ntot * g.batch > ((int64_t)1 << 26)) return;
  if (g.ntot * g.batch / 16 >= ((int64_t)1 << 31)) return;  // lines are counted in 32 bits
  std::vector<int4> tab;
  if (two) {
    const int k = ilog2(g.n[0]), ka = (k + 1) / 2, kb = k - ka;
    // lines of na and nb points; between them e^{2 pi i m / n}, m = 2^kb h + l: the high part
    // is the table of na
    p.fx_off[0] = p.fx_off[2] = 0;
    twiddles(tab, (int64_t)1 << ka, (int64_t)1 << ka);
    p.fx_off[1] = (int64_t)tab.size();
    twiddles(tab, (int64_t)1 << kb, (int64_t)1 << kb);
    p.fx_off[3] = (int64_t)tab.size();
    twiddles(tab, g.n[0], (int64_t)1 << kb);
  } else {
    for (int t = 0; t < g.d; ++t) {
      p.fx_off[t] = -1;
      for (int s = 0; s < t; ++s)
        if (g.n[s] == g.n[t]) p.fx_off[t] = p.fx_off[s];
      if (p.fx_off[t] >= 0) continue;
      p.fx_off[t] = (int64_t)tab.size();
      twiddles(tab, g.n[t], g.n[t]);
    }
  }
  if (plan_malloc(&p.fx_tab, sizeof(int4) * tab.size()) != cudaSuccess ||
      (two && plan_malloc(&p.fx_tmp, sizeof(double2) * (size_t)(g.ntot * g.batch)) != cudaSuccess) ||
      cudaMemcpy(p.fx_tab, tab.data(), sizeof(int4) * tab.size(), cudaMemcpyHostToDevice) != cudaSuccess) {
    cudaGetLastError();
    fft_fix_release(p);
    return;
  }
  p.fx_on = true;
}

template <int TPT>
static cudaError_t launch_pass_t(const FftArgs& a, bool inv, cudaStream_t st) {
  const size_t smem = (size_t)kFftThreads * 4 * TPT * sizeof(I2);
  auto kern = inv ? k_fft<TPT, true> : k_fft<TPT, false>;
  const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return e;
  const int64_t blocks = ((int64_t)a.lines + ((int64_t)1 << a.logC) - 1) >> a.logC;
  kern<<<(unsigned)blocks, kFftThreads, smem, st>>>(a);
  return cudaGetLastError();
}

// Points per CTA: 1024 (16 KB) up to 256-point lines, more where 64-byte segments (four
// neighbouring lines) need them
static cudaError_t launch_pass(FftArgs& a, bool inv, cudaStream_t st) {
  const int tpt = a.logL <= 8 ? 1 : (a.logL == 9 ? 2 : 4);
  a.logC = 10 + (tpt >> 1) - a.logL;  // 1024 tpt points
  if (tpt == 1) return launch_pass_t<1>(a, inv, st);
  if (tpt == 2) return launch_pass_t<2>(a, inv, st);
  return launch_pass_t<4>(a, inv, st);
}

// Roll-off and forward FFT of the coefficients (fhat), or the FFT of the grid in place
// (fhat null), e^-; inv: e^+.
cudaError_t launch_fft_fix(const Plan& p, const void* fhat, void* g, bool inv, cudaStream_t st) {
  const Geom& geo = p.geo;
  const int d = geo.d;
  const bool pad = fhat != nullptr;
  FftArgs a{};
  if (d == 1 && geo.n[0] > kFftMaxL) {
    const int k = ilog2(geo.n[0]), ka = (k + 1) / 2, kb = k - ka;
    a.src = (const double2*)(pad ? fhat : g);
    a.dst = (double2*)p.fx_tmp;
    a.roc = pad ? p.roc_tab : nullptr;
    a.pad = pad;
    a.log_tail = kb;
    a.lead_n = 1;
    a.lines = (uint32_t)geo.batch << kb;
    a.valid = geo.N[0];
    a.logL = ka;
    a.tw = p.fx_tab + p.fx_off[0];
    a.post_hi = p.fx_tab + p.fx_off[2];
    a.post_lo = p.fx_tab + p.fx_off[3];
    a.post_sh = kb;
    a.post_log = k;
    cudaError_t e = launch_pass(a, inv, st);
    if (e != cudaSuccess) return e;
    FftArgs b{};
    b.src = (const double2*)p.fx_tmp;
    b.dst = (double2*)g;
    b.nlead = 1;
    b.lead_n = b.dst_l = (int64_t)1 << ka;
    b.N[0] = b.n[0] = 1u << ka;
    b.lines = (uint32_t)geo.batch << ka;
    b.logL = kb;
    b.tw = p.fx_tab + p.fx_off[1];
    return launch_pass(b, inv, st);
  }
  // padded forward: from the last dimension to the first, so that the leading dimensions
  // still hold coefficients only; in place: any order
  for (int t = d - 1; t >= 0; --t) {
    a = FftArgs{};
    const bool first = pad && t == d - 1;
    a.src = (const double2*)(first ? fhat : g);
    a.dst = (double2*)g;
    a.roc = first ? p.roc_tab : nullptr;
    a.pad = pad;
    for (int s = t + 1; s < d; ++s) a.log_tail += ilog2(geo.n[s]);
    a.nlead = t;
    a.lead_n = 1;
    int64_t lines = (int64_t)geo.batch << a.log_tail;
    for (int s = 0; s < t; ++s) {
      a.N[s] = (uint32_t)(pad ? geo.N[s] : geo.n[s]);
      a.n[s] = (uint32_t)geo.n[s];
      a.lead_n *= geo.n[s];
      lines *= a.N[s];
    }
    a.lines = (uint32_t)lines;
    a.valid = geo.N[t];
    a.logL = ilog2(geo.n[t]);
    a.tw = p.fx_tab + p.fx_off[t];
    const cudaError_t e = launch_pass(a, inv, st);
    if (e != cudaSuccess) return e;
  }
  return cudaSuccess;
}

}  // namespace cg
