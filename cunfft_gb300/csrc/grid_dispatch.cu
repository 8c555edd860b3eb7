// grid_dispatch.cu -- selects the gridding kernel instance for the plan's tap count.
#include <math.h>

#include "kernels_fix.cuh"

namespace cg {

#define CG_DECL(W) cudaError_t grid_launch_w##W(const Plan&, bool, bool, const void*, void*, cudaStream_t);
CG_DECL(4) CG_DECL(6) CG_DECL(8) CG_DECL(10) CG_DECL(12) CG_DECL(14) CG_DECL(16) CG_DECL(18)
CG_DECL(20) CG_DECL(22) CG_DECL(24) CG_DECL(26) CG_DECL(28) CG_DECL(30) CG_DECL(32)
#undef CG_DECL

bool gridding_supported(int d, int W) { return d >= 1 && d <= 3 && W >= 4 && W <= 32 && (W % 2) == 0; }

// Constants of the fixed-point gridding.  vbits: a node's sum is at most 2^vbits times the
// product of the largest tap sums S_t per dimension, which has to stay below 2^63, and each
// sum before the last dimension below 2^59, where its high limb still fits 32 bits with its
// sign (S_t is taken 2 % too large).
FixPar fix_params(const Geom& g) {
  FixPar fp{};
  double all = 0.0, last = 0.0;
  for (int t = 0; t < g.d; ++t) {
    const long double c = 1.0L / (logl(2.0L) * (long double)g.b[t]);
    fp.c60[t] = (uint64_t)llrintl(ldexpl(c, 60));
    fp.c57[t] = (int64_t)llrintl(ldexpl(c, kFixExpFrac));
    fp.es_b2[t] = (double)((long double)g.es_beta[t] / logl(2.0L));
    double most = 0.0;
    for (int i = 0; i <= 16; ++i) {
      double s = 0.0;
      for (int l = 0; l < g.W; ++l) {
        const double y = i / 16.0 + g.m - l, z = 1.0 - y * y * g.es_ia2;
        s += g.window == kWinES ? (z > 0.0 ? exp(g.es_beta[t] * (sqrt(z) - 1.0)) : 0.0) : exp(-y * y / g.b[t]);
      }
      most = s > most ? s : most;
    }
    last = log2(1.02 * most);  // between the sampled fractions the sum hardly moves
    all += last;
  }
  const int a = (int)floor(63.0 - all), b = (int)floor(59.0 - (all - last));
  fp.vbits = a < b ? a : b;
  if (fp.vbits > 55) fp.vbits = 55;
  return fp;
}

// Larger of the interpolation and spreading kernels' shared-memory needs.
size_t gridding_smem_bytes(const Plan& p) {
  const int d = p.geo.d, W = p.geo.W;
  if (p.prec == kF64) {
    if (d == 3 && W > kFixWholeW) return 0;  // the planes go through in slabs
    const size_t a = fix_smem_bytes(d, W, p.tl.E[0], false), b = fix_smem_bytes(d, W, p.tl.E[0], true);
    return a > b ? a : b;
  }
  const size_t real = 4;
  const int nwarps = p.tl.threads / 32;
  const size_t a = grid_extra_smem(d, W, real, nwarps, p.tl.smem_tile, false);
  const size_t b = grid_extra_smem(d, W, real, nwarps, p.tl.smem_tile, true);
  return p.tl.smem_tile + (a > b ? a : b);
}

static cudaError_t dispatch(const Plan& p, bool spread, bool alone, const void* in, void* out, cudaStream_t st) {
  if (spread && p.tl.spread_kernel == CUNFFT_X_SPREAD_TENSOR) return grid_launch_spread_tc(p, in, out, st);
  if (!spread && p.tl.interp_kernel == CUNFFT_X_INTERP_TENSOR) return grid_launch_interp_tc(p, in, out, st);
  if (spread && p.tl.spread_kernel == CUNFFT_X_SPREAD_REGISTER) return grid_launch_spread_reg(p, in, out, st);
  switch (p.geo.W) {
#define CG_CASE(W) case W: return grid_launch_w##W(p, spread, alone, in, out, st);
    CG_CASE(4) CG_CASE(6) CG_CASE(8) CG_CASE(10) CG_CASE(12) CG_CASE(14) CG_CASE(16) CG_CASE(18)
    CG_CASE(20) CG_CASE(22) CG_CASE(24) CG_CASE(26) CG_CASE(28) CG_CASE(30) CG_CASE(32)
#undef CG_CASE
    default: return cudaErrorInvalidValue;
  }
}

cudaError_t launch_interp(const Plan& p, const void* g, void* f, bool alone, cudaStream_t st) {
  if (p.bins.M == 0) return cudaSuccess;
  cudaError_t e = cudaMemsetAsync(p.bins.work, 0, sizeof(int32_t), st);
  if (e != cudaSuccess) return e;
  return dispatch(p, false, alone, g, f, st);
}

cudaError_t launch_spread(const Plan& p, const void* f, void* g, bool alone, cudaStream_t st) {
  if (p.bins.M == 0) return cudaSuccess;
  cudaError_t e = cudaMemsetAsync(p.bins.work + 1, 0, sizeof(int32_t), st);
  if (e != cudaSuccess) return e;
  return dispatch(p, true, alone, f, g, st);
}

}  // namespace cg
