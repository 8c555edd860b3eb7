// kernels_grad_tile.cuh -- node-position gradient of the FP32 form on staged tiles.
//
// The sums of kernels_grad.cu in the same order and rounding (one thread per node, outer
// dimension outermost), on the work items and tiles of the shared-tile interpolation: the
// node's window comes from shared memory, where the scattered reads of a warp cost a few
// wavefronts instead of up to 32 cache lines, and the taps w and const y w are formed in
// integers (fixmath.h) and rounded to FP32 once, as FP64 taps would be, instead of FP64
// exponentials.
// Bound: shared-memory wavefronts of scattered reads (about seven for a warp's 32 windows), the
// FP64 pipe (coordinates) and the integer multiply-adds (taps) close to one another.
// 2D, m = 6, M = 2^18: 92 us; gathers from global memory and FP64 taps before: 400 us.
#pragma once

#include "kernels_fix.cuh"

namespace cg {

constexpr int kGradThreads = 128;

// Constants of the derivative taps: dw = c y w with c = -2 n / b (Gaussian), as a 63-bit
// mantissa and a power of two.
struct GradPar {
  uint64_t mant[kMaxDim];  // |c| = mant 2^-63 2^e, mant in [2^62, 2^63)
  float scale[kMaxDim];    // 2^e / 2^60, negative
};

// Gradient of one node (coordinates x) on its instance's grid, through global memory.
template <typename T>
__device__ __forceinline__ void grad_node_global(const double* __restrict__ x, const typename Cx<T>::t* __restrict__ gi,
                                              typename Cx<T>::t gf, double* __restrict__ out, const Geom& geo) {
  using C = typename Cx<T>::t;
  const int d = geo.d, W = geo.W;
  T w[kMaxDim][kMaxTaps], dw[kMaxDim][kMaxTaps];
  int64_t u[kMaxDim] = {0, 0, 0};
  for (int t = 0; t < d; ++t) {
    const double xt = x[t];
    const double nx = __dmul_rn(xt, (double)geo.n[t]);
    u[t] = (int64_t)__double2ll_rn(nx) - (signbit(xt) ? 1 : 0) - geo.m;
    const double c = __dsub_rn(nx, (double)u[t]);
    if (geo.window == kWinES) {
      // phi = exp(beta (s - 1)), s = sqrt(1 - y^2/alpha^2); dphi/dy = -phi beta y / (alpha^2 s)
      const double beta = geo.es_beta[t];
      for (int l = 0; l < W; ++l) {
        const double y = c - (double)l, z = 1.0 - (y * y) * geo.es_ia2;
        const double s = z > 0.0 ? sqrt(z) : 0.0;
        const double e = z > 0.0 ? exp(beta * (s - 1.0)) : 0.0;
        w[t][l] = (T)e;
        dw[t][l] = z > 0.0 ? (T)(-e * beta * y * geo.es_ia2 / s * (double)geo.n[t]) : (T)0;
      }
    } else {
      const double ib = 1.0 / geo.b[t];
      for (int l = 0; l < W; ++l) {
        const double y = c - (double)l;
        const double e = exp(-(y * y) * ib);
        w[t][l] = (T)e;
        dw[t][l] = (T)(-2.0 * y * ib * e * (double)geo.n[t]);
      }
    }
  }
  for (int t = d; t < kMaxDim; ++t) {
    w[t][0] = (T)1;
    dw[t][0] = (T)0;
  }
  const int W1 = d >= 2 ? W : 1, W2 = d >= 3 ? W : 1;
  // partial sums: p[t] = sum g * (derivative in dim t, plain weights elsewhere)
  T pr[kMaxDim] = {0, 0, 0}, pi[kMaxDim] = {0, 0, 0};
  for (int l0 = 0; l0 < W; ++l0) {
    const int64_t i0 = wrap_n(u[0] + l0, geo.n[0]);
    for (int l1 = 0; l1 < W1; ++l1) {
      const int64_t i1 = d >= 2 ? wrap_n(u[1] + l1, geo.n[1]) : 0;
      // inner sums over the last dimension: plain and derivative weights
      T ar = 0, ai = 0, br = 0, bi = 0;
      for (int l2 = 0; l2 < W2; ++l2) {
        const int64_t i2 = d >= 3 ? wrap_n(u[2] + l2, geo.n[2]) : 0;
        int64_t gidx = i0;
        if (d >= 2) gidx = gidx * geo.n[1] + i1;
        if (d >= 3) gidx = gidx * geo.n[2] + i2;
        const C v = gi[gidx];
        const T a = d >= 3 ? w[2][l2] : (T)1, b = d >= 3 ? dw[2][l2] : (T)0;
        ar += a * v.x; ai += a * v.y;
        br += b * v.x; bi += b * v.y;
      }
      // (ar, ai): plain in last dim; (br, bi): derivative in dim 2
      const T w1 = d >= 2 ? w[1][l1] : (T)1, dw1 = d >= 2 ? dw[1][l1] : (T)0;
      const T w0 = w[0][l0], dw0 = dw[0][l0];
      pr[0] += dw0 * w1 * ar; pi[0] += dw0 * w1 * ai;
      if (d >= 2) { pr[1] += w0 * dw1 * ar; pi[1] += w0 * dw1 * ai; }
      if (d >= 3) { pr[2] += w0 * w1 * br; pi[2] += w0 * w1 * bi; }
    }
  }
  for (int t = 0; t < d; ++t) out[t] = geo.norm * ((double)gf.x * (double)pr[t] + (double)gf.y * (double)pi[t]);
}

// ... out of line, for the few nodes of a tile that need it
static __device__ __noinline__ void grad_node_moved(const double* __restrict__ x, const float2* __restrict__ gi, float2 gf,
                                                    double* __restrict__ out, const Geom& geo) {
  grad_node_global<float>(x, gi, gf, out, geo);
}

template <int D, int W>
__global__ void __launch_bounds__(kGradThreads)
    k_grad_tile(const double* __restrict__ x, const float2* __restrict__ g, const float2* __restrict__ grad_f,
                double* __restrict__ grad_x, Geom geo, Tiling tl, Bins bins, FixPar fp, GradPar gp) {
  constexpr int SH = off_bits(D);
  constexpr uint32_t MASK = (1u << SH) - 1u;
  constexpr int S = fixed_row_stride(D, W), PS = fixed_plane_stride(D, W);
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ int4 cur;
  float2* tile = reinterpret_cast<float2*>(smem);
  uint64_t* tab = reinterpret_cast<uint64_t*>(smem + tl.smem_tile);
  for (int i = threadIdx.x; i < kFixExpTab; i += blockDim.x) tab[i] = fix_exp_entry(i);

  while (next_item(bins, 0, &cur)) {
    const int4 item = cur;
    const TileOrigin o = decode_tile<D>(geo, tl, item.x);
    load_tile<D, W, float2>(tile, g + o.inst * geo.ntot, geo, tl, o, 0, tl.E[0]);
    __syncthreads();
    for (int k = item.y + threadIdx.x; k < item.z; k += kGradThreads) {
      const int j = bins.sidx[k];
      const uint32_t off = (uint32_t)bins.soff[k];
      float w[D][W], dw[D][W];
      bool moved = false;
#pragma unroll
      for (int t = 0; t < D; ++t) {
        const double xt = x[(int64_t)j * D + t], n = (double)geo.n[t];
        const double nx = __dmul_rn(xt, n);
        const int64_t u = __double2ll_rn(nx) - (signbit(xt) ? 1 : 0);
        const double fr = __dsub_rn(nx, (double)u);
        const bool finite = fabs(fr) < 2.0;
        int64_t s = u - geo.m;  // window start, as the binning found it unless x has changed since
        if (s < 0) s += geo.n[t];
        if (s < 0 || s >= geo.n[t]) s = wrap_n(s, geo.n[t]);
        moved |= finite && s != o.a[t] + ((off >> (SH * t)) & MASK);
        if (!finite) {
          for (int l = 0; l < W; ++l) w[t][l] = dw[t][l] = __int_as_float(0x7fc00000);
        } else if (geo.window == kWinES) {
          for (int l = 0; l < W; ++l) {
            const double y = fr + (double)(geo.m - l), z = 1.0 - (y * y) * geo.es_ia2;
            const double s = z > 0.0 ? sqrt(z) : 0.0, e = z > 0.0 ? exp(geo.es_beta[t] * (s - 1.0)) : 0.0;
            w[t][l] = (float)e;
            dw[t][l] = z > 0.0 ? (float)(-e * geo.es_beta[t] * y * geo.es_ia2 / s * n) : 0.f;
          }
        } else {
          const FixGauss pq = fix_stage(geo, fp, t, fr);
          const int64_t y0 = __double2ll_rn(fr * 288230376151711744.0) + ((int64_t)geo.m << 58);  // units of 2^-58
#pragma unroll 2
          for (int l = 0; l < W; ++l) {
            const int kk = geo.m - l;
            const int64_t tap = fix_gauss_tap<62>(pq, kk, (int64_t)(kk * kk) * fp.c57[t], tab);
            w[t][l] = __ll2float_rn(tap) * 2.168404344971009e-19f;  // 2^-62
            const int64_t y = y0 - ((int64_t)l << 58);
            const uint64_t wy = fix_mulhi64((uint64_t)tap << 1, (uint64_t)(y < 0 ? -y : y));   // w |y| in units of 2^-57
            const float d = __ll2float_rn((int64_t)fix_mulhi64(wy << 4, gp.mant[t])) * gp.scale[t];
            dw[t][l] = y < 0 ? -d : d;
          }
        }
      }
      if (moved) {  // another window than the tile's: the coordinates count, as in the other form
        grad_node_moved(x + (int64_t)j * D, g + o.inst * geo.ntot, grad_f[j], grad_x + (int64_t)j * D, geo);
        continue;
      }
      float pr[D], pi[D], wl[W], dl[W];
#pragma unroll
      for (int t = 0; t < D; ++t) pr[t] = pi[t] = 0.f;
#pragma unroll
      for (int l = 0; l < W; ++l) {
        wl[l] = w[D - 1][l];
        dl[l] = dw[D - 1][l];
      }
      if constexpr (D == 1) {
        const float2* tb = tile + (off & MASK);
#pragma unroll
        for (int l = 0; l < W; ++l) {
          const float2 v = tb[l];
          pr[0] = __fmaf_rn(dl[l], v.x, pr[0]);
          pi[0] = __fmaf_rn(dl[l], v.y, pi[0]);
        }
      } else if constexpr (D == 2) {
        const float2* tb = tile + (int)(off & MASK) * S + (int)((off >> SH) & MASK);
#pragma unroll 1
        for (int l0 = 0; l0 < W; ++l0, tb += S) {
          const float w0 = w[0][l0], d0 = dw[0][l0];
#pragma unroll
          for (int l = 0; l < W; ++l) {
            const float2 v = tb[l];
            const float a = __fmul_rn(d0, wl[l]), b = __fmul_rn(w0, dl[l]);
            pr[0] = __fmaf_rn(a, v.x, pr[0]);
            pi[0] = __fmaf_rn(a, v.y, pi[0]);
            pr[1] = __fmaf_rn(b, v.x, pr[1]);
            pi[1] = __fmaf_rn(b, v.y, pi[1]);
          }
        }
      } else {
        const float2* tb0 = tile + (int)(off & MASK) * PS + (int)((off >> SH) & MASK) * S + (int)(off >> (2 * SH));
#pragma unroll 1
        for (int l0 = 0; l0 < W; ++l0) {
          const float w0 = w[0][l0], d0 = dw[0][l0];
#pragma unroll 1
          for (int l1 = 0; l1 < W; ++l1) {
            const float2* tb = tb0 + l0 * PS + l1 * S;
            float ar = 0.f, ai = 0.f, br = 0.f, bi = 0.f;
#pragma unroll
            for (int l = 0; l < W; ++l) {
              const float2 v = tb[l];
              ar = __fmaf_rn(wl[l], v.x, ar);
              ai = __fmaf_rn(wl[l], v.y, ai);
              br = __fmaf_rn(dl[l], v.x, br);
              bi = __fmaf_rn(dl[l], v.y, bi);
            }
            const float w1 = w[1][l1], d1 = dw[1][l1];
            const float a = __fmul_rn(d0, w1), b = __fmul_rn(w0, d1), c = __fmul_rn(w0, w1);
            pr[0] = __fmaf_rn(a, ar, pr[0]);
            pi[0] = __fmaf_rn(a, ai, pi[0]);
            pr[1] = __fmaf_rn(b, ar, pr[1]);
            pi[1] = __fmaf_rn(b, ai, pi[1]);
            pr[2] = __fmaf_rn(c, br, pr[2]);
            pi[2] = __fmaf_rn(c, bi, pi[2]);
          }
        }
      }
      const float2 gf = grad_f[j];
#pragma unroll
      for (int t = 0; t < D; ++t)
        grad_x[(int64_t)j * D + t] = geo.norm * ((double)gf.x * (double)pr[t] + (double)gf.y * (double)pi[t]);
    }
    __syncthreads();
  }
}

}  // namespace cg
