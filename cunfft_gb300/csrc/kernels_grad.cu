// kernels_grad.cu -- node-position gradient of the forward NFFT (derivative-of-window gridding).
//
// f_j = sum_l g[u + l] prod_t psi_t(c_t - l_t),  c_t = n_t x_t - u_t, so
//   d f_j / d x_{j,t} = n_t sum_l g[u + l] psi_t'(c_t - l_t) prod_{s != t} psi_s(c_s - l_s),
//   Gaussian psi(y) = K exp(-y^2/b): psi'(y) = -(2 y / b) psi(y);
//   ES psi(y) = exp(beta (s - 1)), s = sqrt(1 - y^2/alpha^2): psi'(y) = -psi(y) beta y / (alpha^2 s).
// The kernel evaluates the d partial derivatives on the same roll-off-corrected,
// FFT'd grid g as the forward transform and contracts them with the incoming
// gradient: grad_x[j, t] = Re(conj(grad_f_j) * d f_j / d x_{j,t}).
// No reference counterpart (the reference has no differentiable transform).
// FP64 node reduction and weights; accumulation in the plan's real type.  The FP32 form runs
// on staged tiles (kernels_grad_tile.cuh); the kernel here, one thread per node with the
// grid read through L1/L2, takes the FP64 form and 3D windows wider than 16 taps.
#include <math.h>

#include "kernels_grad_tile.cuh"

namespace cg {

template <typename T>
__global__ void __launch_bounds__(128) k_interp_grad(const double* __restrict__ x,
                                                     const typename Cx<T>::t* __restrict__ g,
                                                     const typename Cx<T>::t* __restrict__ grad_f,
                                                     double* __restrict__ grad_x, Geom geo,
                                                     const int32_t* __restrict__ inst_off, int64_t M) {
  const int d = geo.d;
  for (int64_t j = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; j < M; j += (int64_t)gridDim.x * blockDim.x) {
    int inst = 0;
    if (geo.batch > 1) {
      int lo = 0, hi = geo.batch;
      while (hi - lo > 1) {
        const int mid = (lo + hi) >> 1;
        if (inst_off[mid] <= j) lo = mid; else hi = mid;
      }
      inst = lo;
    }
    grad_node_global<T>(x + j * d, g + (int64_t)inst * geo.ntot, grad_f[j], grad_x + j * d, geo);
  }
}

#define CG_DECL(W) \
  cudaError_t grid_grad_w##W(const Plan&, const GradPar&, const void*, const void*, double*, cudaStream_t);
CG_DECL(4) CG_DECL(6) CG_DECL(8) CG_DECL(10) CG_DECL(12) CG_DECL(14) CG_DECL(16) CG_DECL(18)
CG_DECL(20) CG_DECL(22) CG_DECL(24) CG_DECL(26) CG_DECL(28) CG_DECL(30) CG_DECL(32)
#undef CG_DECL

static cudaError_t launch_grad_tile(const Plan& p, const void* g, const void* grad_f, double* grad_x, cudaStream_t st) {
  GradPar gp{};
  for (int t = 0; t < p.geo.d; ++t) {
    int e;
    const double f = frexp(2.0 / p.geo.b[t] * (double)p.geo.n[t], &e);  // f in [1/2, 1)
    gp.mant[t] = (uint64_t)ldexp(f, 63);
    gp.scale[t] = -(float)ldexp(1.0, e - 60);  // the kernel's product: w |y| 2^61 f 2^63 / 2^64
  }
  const cudaError_t e = cudaMemsetAsync(p.bins.work, 0, sizeof(int32_t), st);
  if (e != cudaSuccess) return e;
  switch (p.geo.W) {
#define CG_CASE(W) case W: return grid_grad_w##W(p, gp, g, grad_f, grad_x, st);
    CG_CASE(4) CG_CASE(6) CG_CASE(8) CG_CASE(10) CG_CASE(12) CG_CASE(14) CG_CASE(16) CG_CASE(18)
    CG_CASE(20) CG_CASE(22) CG_CASE(24) CG_CASE(26) CG_CASE(28) CG_CASE(30) CG_CASE(32)
#undef CG_CASE
    default: return cudaErrorInvalidValue;
  }
}

cudaError_t launch_interp_grad(const Plan& p, const void* g, const void* grad_f, double* grad_x, cudaStream_t st) {
  if (p.M == 0) return cudaSuccess;
  // FP32 on staged tiles, in 3D up to 16 taps: above, the 6 W taps of a thread live in local memory
  // (3D n = 128^3, 5e4 nodes, tile / thread per node: W = 16 0.92 / 1.07 ms, W = 18 3.5 / 1.5 ms,
  // W = 24 37 / 3.2 ms; 2D n = 512^2, 1e5 nodes, W = 26 0.14 / 0.46 ms).  The shared-tile kernels'
  // shared memory covers the tile and more than the exponential's table.
  if (p.prec == kF32 && (p.geo.d < 3 || p.geo.W <= 16)) return launch_grad_tile(p, g, grad_f, grad_x, st);
  int64_t b = (p.M + 127) / 128;
  if (b > (int64_t)p.num_sms * 16) b = (int64_t)p.num_sms * 16;
  if (p.prec == kF64)
    k_interp_grad<double><<<(unsigned)b, 128, 0, st>>>(p.x, (const double2*)g, (const double2*)grad_f, grad_x, p.geo,
                                                       p.bins.inst_off, p.M);
  else
    k_interp_grad<float><<<(unsigned)b, 128, 0, st>>>(p.x, (const float2*)g, (const float2*)grad_f, grad_x, p.geo,
                                                      p.bins.inst_off, p.M);
  return cudaGetLastError();
}

}  // namespace cg
