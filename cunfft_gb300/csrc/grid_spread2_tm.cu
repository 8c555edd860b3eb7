// grid_spread2_tm.cu -- launcher of the 2D FP32 tensor-core spreading kernel
// (kernels_spread2_tm.cuh).
#include <algorithm>

#include "kernels_spread2_sub.cuh"
#include "kernels_spread2_tm.cuh"

namespace cg {

bool spread2_tm_supported(const Plan& p) {
  return p.prec == kF32 && spread2_tm_ok(p.geo.d, p.geo.W, p.tl.T[0], p.tl.T[1]);
}

// The kernel allocates all 512 tensor-memory columns; its dynamic shared memory is at
// least half of the SM's 228 KB, so that two CTAs never share an SM and tcgen05.alloc
// never waits.
static constexpr size_t kT2SmemFloor = 228u * 1024u / 2u + 1u;

// The sub-tile kernel, where the binning makes its items.  Its items cost about as much with
// few nodes as with many, so a grid of many sub-tiles with only a few nodes each goes to the
// whole-tile kernel.  Measured (m = 6; us, sub-tile / whole-tile): n = 1024^2 (4096 sub-tiles)
// M = 1000 13 / 19, 10^4 28 / 22, 5 10^4 30 / 33, 2 10^5 37 / 83; n = 256^2 M = 1000 11 / 19,
// 2 10^5 28 / 76.
static bool use_sub(const Plan& p) {
  if (!p.tl.sub_on || !p.tl.sub_items) return false;
  const int64_t keys = p.tl.tiles_total * p.tl.ns;
  return p.bins.M >= 8 * keys || std::min(p.bins.M, keys) <= (int64_t)2 * p.num_sms * kS2PerSm;
}

template <int W>
static cudaError_t launch_sub(const Plan& p, const void* in, void* out, cudaStream_t st) {
  auto kern = p.geo.window == kWinES ? k_spread2_sub<W, kWinES> : k_spread2_sub<W, kWinGauss>;
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kS2Smem);
  if (e != cudaSuccess) return e;
  // (the occupancy call counts one CTA per SM for a kernel that allocates tensor memory)
  kern<<<p.num_sms * kS2PerSm, kS2Threads, kS2Smem, st>>>((const float2*)in, (float2*)out, p.geo, p.tl, p.bins);
  return cudaGetLastError();
}

template <int W>
static cudaError_t launch_t2(const Plan& p, const void* in, void* out, cudaStream_t st) {
  if (!spread2_tm_supported(p)) return cudaErrorInvalidConfiguration;
  if (use_sub(p)) return launch_sub<W>(p, in, out, st);
  const size_t smem = std::max<size_t>(t2_layout().total, kT2SmemFloor);
  auto kern = p.geo.window == kWinES ? k_spread2_tm<W, kWinES> : k_spread2_tm<W, kWinGauss>;
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return e;
  int per_sm = 0;
  e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, kT2Threads, smem);
  if (e != cudaSuccess) return e;
  if (per_sm != 1) return cudaErrorInvalidConfiguration;
  e = spread_tc_permute(p, in, st);
  if (e != cudaSuccess) return e;
  kern<<<p.num_sms, kT2Threads, smem, st>>>((const float2*)in, (float2*)out, p.geo, p.tl, p.bins);
  return cudaGetLastError();
}

cudaError_t grid_launch_spread2_tm(const Plan& p, const void* in, void* out, cudaStream_t st) {
  switch (p.geo.W) {
    case 4: return launch_t2<4>(p, in, out, st);
    case 6: return launch_t2<6>(p, in, out, st);
    case 8: return launch_t2<8>(p, in, out, st);
    case 10: return launch_t2<10>(p, in, out, st);
    case 12: return launch_t2<12>(p, in, out, st);
    case 14: return launch_t2<14>(p, in, out, st);
    case 16: return launch_t2<16>(p, in, out, st);
    default: return cudaErrorInvalidValue;
  }
}

}  // namespace cg
