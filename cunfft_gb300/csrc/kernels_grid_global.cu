// kernels_grid_global.cu -- gridding without a shared-memory tile.
//
// Used by the FP32 form when the padded tile of even a single grid cell does not fit in
// the 227 KB of shared memory a CTA may use: the widest windows in 3D.  Same work items as the tiled kernels;
// one thread per node, taps read from (interpolation) or atomically added to
// (spreading) the oversampled grid in global memory, weights in the plan's real
// type from the binned fractions.  Results agree with the tiled kernels.
#include "kernels_grid.cuh"

namespace cg {

template <int D, typename T, bool SPREAD>
__global__ void __launch_bounds__(128) k_grid_global(const typename Cx<T>::t* __restrict__ in,
                                                     typename Cx<T>::t* __restrict__ out, Geom geo, Tiling tl,
                                                     Bins bins) {
  using C = typename Cx<T>::t;
  __shared__ int4 cur;
  const T* sfrac = reinterpret_cast<const T*>(bins.sfrac);
  while (next_item(bins, SPREAD ? 1 : 0, &cur)) {
    const int4 item = cur;
    const TileOrigin o = decode_tile<D>(geo, tl, item.x);
    for (int64_t k = item.y + threadIdx.x; k < item.z; k += blockDim.x) {
      grid_node_global<D, T, SPREAD>(in, out, geo, o, bins.sidx[k], (uint32_t)bins.soff[k], sfrac + k * D);
    }
    __syncthreads();
  }
}

template <int D, typename T, bool SPREAD>
static cudaError_t launch_global(const Plan& p, const void* in, void* out, cudaStream_t st) {
  using C = typename Cx<T>::t;
  auto kern = k_grid_global<D, T, SPREAD>;
  int per_sm = 0;
  cudaError_t e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, 128, 0);
  if (e != cudaSuccess) return e;
  kern<<<p.num_sms * (per_sm > 0 ? per_sm : 1), 128, 0, st>>>((const C*)in, (C*)out, p.geo, p.tl, p.bins);
  return cudaGetLastError();
}

cudaError_t grid_launch_global(const Plan& p, bool spread, const void* in, void* out, cudaStream_t st) {
  const int d = p.geo.d;
  if (d == 1) return spread ? launch_global<1, float, true>(p, in, out, st) : launch_global<1, float, false>(p, in, out, st);
  if (d == 2) return spread ? launch_global<2, float, true>(p, in, out, st) : launch_global<2, float, false>(p, in, out, st);
  return spread ? launch_global<3, float, true>(p, in, out, st) : launch_global<3, float, false>(p, in, out, st);
}

}  // namespace cg
