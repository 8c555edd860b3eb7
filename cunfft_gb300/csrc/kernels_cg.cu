// kernels_cg.cu -- vector algebra of conjugate gradients on the normal equations
// (A^H W A + lam I) x = b, between the plan's forward and adjoint transforms.
//
// Three launches per iteration on the plan's stream, every scalar in device memory, so that
// the host neither waits for a dot product nor launches one kernel per vector operation:
//   dot     ap += lam p,          pap[i] = Re <p, ap>
//   step    x += alpha p, r -= alpha ap, alpha = rr[i] / pap[i],     rr[i + 1] = <r, r>
//   turn    p = r + (rr[i + 1] / rr[i]) p, hist[i] = sqrt(rr[i + 1] / bb), stop[i + 1]
// Sums in FP64 (the scalars as well), vectors in the plan's real type.  An iteration whose
// predecessor reached the tolerance changes nothing.
// Bound: HBM or, for the usual small vectors, launch latency.  N = 192^2, M = 150001, ten
// iterations: 1.81 ms; with one library kernel per operation and a host wait per iteration
// before: 2.97 ms.
#include "runtime.h"

namespace cg {

constexpr int kCgThreads = 256;

// the CTA's sum added to *out
__device__ __forceinline__ void cg_add(double v, double* out) {
  __shared__ double s[kCgThreads / 32];
  for (int o = 16; o >= 1; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  if ((threadIdx.x & 31) == 0) s[threadIdx.x >> 5] = v;
  __syncthreads();
  if (threadIdx.x < 32) {
    v = threadIdx.x < kCgThreads / 32 ? s[threadIdx.x] : 0.0;
    for (int o = 4; o >= 1; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    if (threadIdx.x == 0) atomicAdd(out, v);
  }
  __syncthreads();
}

// scalars: bb, rr[iters + 1], pap[iters], hist[iters]
struct CgScal {
  double* base;
  int64_t iters;
  __device__ double* bb() const { return base; }
  __device__ double* rr(int64_t i) const { return base + 1 + i; }
  __device__ double* pap(int64_t i) const { return base + 2 + iters + i; }
  __device__ double* hist(int64_t i) const { return base + 2 + 2 * iters + i; }
};

template <typename T>
__global__ void __launch_bounds__(kCgThreads) k_cg_begin(const typename Cx<T>::t* __restrict__ b,
                                                         const typename Cx<T>::t* __restrict__ r, int64_t n, CgScal sc) {
  double bb = 0.0, rr = 0.0;
  for (int64_t i = blockIdx.x * (int64_t)kCgThreads + threadIdx.x; i < n; i += (int64_t)gridDim.x * kCgThreads) {
    bb += (double)b[i].x * b[i].x + (double)b[i].y * b[i].y;
    rr += (double)r[i].x * r[i].x + (double)r[i].y * r[i].y;
  }
  cg_add(bb, sc.bb());
  cg_add(rr, sc.rr(0));
}

template <typename T>
__global__ void __launch_bounds__(kCgThreads) k_cg_dot(const typename Cx<T>::t* __restrict__ p,
                                                       typename Cx<T>::t* __restrict__ ap, int64_t n, T lam, int64_t it,
                                                       CgScal sc, const int32_t* __restrict__ stop) {
  if (stop[it]) return;
  double s = 0.0;
  for (int64_t i = blockIdx.x * (int64_t)kCgThreads + threadIdx.x; i < n; i += (int64_t)gridDim.x * kCgThreads) {
    const typename Cx<T>::t v = p[i];
    typename Cx<T>::t a = ap[i];
    if (lam != (T)0) {
      a.x += lam * v.x;
      a.y += lam * v.y;
      ap[i] = a;
    }
    s += (double)v.x * a.x + (double)v.y * a.y;
  }
  cg_add(s, sc.pap(it));
}

template <typename T>
__global__ void __launch_bounds__(kCgThreads) k_cg_step(typename Cx<T>::t* __restrict__ x, typename Cx<T>::t* __restrict__ r,
                                                        const typename Cx<T>::t* __restrict__ p,
                                                        const typename Cx<T>::t* __restrict__ ap, int64_t n, int64_t it,
                                                        CgScal sc, const int32_t* __restrict__ stop) {
  if (stop[it]) return;
  const T alpha = (T)(*sc.rr(it) / *sc.pap(it));
  double s = 0.0;
  for (int64_t i = blockIdx.x * (int64_t)kCgThreads + threadIdx.x; i < n; i += (int64_t)gridDim.x * kCgThreads) {
    const typename Cx<T>::t pi = p[i], ai = ap[i];
    typename Cx<T>::t xi = x[i], ri = r[i];
    xi.x += alpha * pi.x;
    xi.y += alpha * pi.y;
    ri.x -= alpha * ai.x;
    ri.y -= alpha * ai.y;
    x[i] = xi;
    r[i] = ri;
    s += (double)ri.x * ri.x + (double)ri.y * ri.y;
  }
  cg_add(s, sc.rr(it + 1));
}

template <typename T>
__global__ void __launch_bounds__(kCgThreads) k_cg_turn(const typename Cx<T>::t* __restrict__ r,
                                                        typename Cx<T>::t* __restrict__ p, int64_t n, int64_t it, double tol,
                                                        CgScal sc, int32_t* __restrict__ stop) {
  if (stop[it]) {
    if (blockIdx.x == 0 && threadIdx.x == 0) stop[it + 1] = 1;
    return;
  }
  const double rr = *sc.rr(it + 1);
  const T beta = (T)(rr / *sc.rr(it));
  for (int64_t i = blockIdx.x * (int64_t)kCgThreads + threadIdx.x; i < n; i += (int64_t)gridDim.x * kCgThreads) {
    const typename Cx<T>::t ri = r[i];
    typename Cx<T>::t pi = p[i];
    pi.x = ri.x + beta * pi.x;
    pi.y = ri.y + beta * pi.y;
    p[i] = pi;
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    const double rel = sqrt(rr) / sqrt(*sc.bb());
    *sc.hist(it) = rel;
    stop[it + 1] = rel <= tol ? 1 : 0;
  }
}

template <typename T>
static void launch_cg_t(int stage, int blocks, int64_t n, int64_t it, double lam, double tol, const void* b, void* x, void* r,
                        void* p, void* ap, CgScal sc, int32_t* stop, cudaStream_t st) {
  using C = typename Cx<T>::t;
  if (stage == CUNFFT_X_CG_BEGIN) k_cg_begin<T><<<blocks, kCgThreads, 0, st>>>((const C*)b, (const C*)r, n, sc);
  if (stage == CUNFFT_X_CG_DOT) k_cg_dot<T><<<blocks, kCgThreads, 0, st>>>((const C*)p, (C*)ap, n, (T)lam, it, sc, stop);
  if (stage == CUNFFT_X_CG_STEP)
    k_cg_step<T><<<blocks, kCgThreads, 0, st>>>((C*)x, (C*)r, (const C*)p, (const C*)ap, n, it, sc, stop);
  if (stage == CUNFFT_X_CG_TURN) k_cg_turn<T><<<blocks, kCgThreads, 0, st>>>((const C*)r, (C*)p, n, it, tol, sc, stop);
}

cudaError_t launch_cg(const Plan& p, int stage, int64_t it, int64_t iters, double lam, double tol, const void* b, void* x,
                      void* r, void* pv, void* ap, double* scal, int32_t* stop, cudaStream_t st) {
  const int64_t n = p.geo.Ntot * p.geo.batch;
  int64_t blocks = (n + kCgThreads - 1) / kCgThreads;
  if (blocks > (int64_t)p.num_sms * 4) blocks = (int64_t)p.num_sms * 4;
  const CgScal sc{scal, iters};
  if (p.prec == kF64) launch_cg_t<double>(stage, (int)blocks, n, it, lam, tol, b, x, r, pv, ap, sc, stop, st);
  else launch_cg_t<float>(stage, (int)blocks, n, it, lam, tol, b, x, r, pv, ap, sc, stop, st);
  return cudaGetLastError();
}

}  // namespace cg
