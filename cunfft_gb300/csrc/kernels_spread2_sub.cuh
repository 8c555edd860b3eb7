// kernels_spread2_sub.cuh -- 2D FP32 spreading on the tensor cores, by 16 x 16 sub-tiles.
//
// The binning orders a tile's nodes by 16 x 16 sub-tile of window starts and makes items of
// at most 128 nodes of one sub-tile (for the 2D interpolation).  An item's nodes reach only
// 16 + W - 1 <= 31 grid rows and columns, so its part of the grid is a small product over
// its nodes,
//     D[c 32 + p1, p0] = sum_j (w1_j[p1 - o1_j] f_j^c s) (w0_j[p0 - o0_j] 2^10),   c = Re, Im,
// M = 128 rows: the FP16 hi parts of the 64 left rows above their lo parts, N = 32 columns,
// with the right factors' hi and lo parts one after the other: two MMAs per 16 nodes give
// all four hi / lo products, and the lo half is added to the hi half on the way out.
// s = 2^(14 - e) with 2^e above the item's largest sample, so no pass over the samples goes
// first and no permuted copy is made.
//
// A CTA of 128 threads takes items with the grid's stride: it loads the nodes (thread =
// node, the next item's one item ahead), then builds operands 32 nodes at a time into two
// stages (thread = two nodes by every eighth row; the two nodes' values are one word of the
// operand and the leading stride of 160 bytes keeps a warp's words in different banks), one
// thread issues the MMAs, and the 32 x 64 sums leave tensor memory through a staging row
// per grid row as bulk FP32 reductions.  Several CTAs per SM overlap one's loads, MMAs and
// reductions with another's tap arithmetic.  Every mbarrier wait is bounded; one that gives
// up sets the device status flag and the CTA leaves.
//
// Against the whole-tile kernel (kernels_spread2_tm.cuh), whose operands cover the tile's 77
// rows and columns for every node and whose items add out 77 x 77 cells: batched 2D (64 x
// 256^2, m = 5, 6.77M nodes) 0.83 ms, there 1.66 ms and 0.05 ms for the permuted samples;
// clustered (N = 512^2, m = 6, 786K nodes) 84 us, there 205 and 16.  Bound: instruction issue
// (57 % of slots with 20 warps per SM: exponentials, FP16 splits) and the CTA's barriers.
#pragma once

#include "kernels_interp2_tc.cuh"
#include "kernels_spread_tc.cuh"

namespace cg {

constexpr int kS2Threads = 128;
constexpr int kS2Chunk = 32;               // nodes per operand stage
constexpr uint32_t kS2LBO = 160;           // core matrices along K
constexpr uint32_t kS2SBO = (kS2Chunk / 8) * kS2LBO;
constexpr uint32_t kS2ABytes = 16 * kS2SBO;  // 128 rows
constexpr uint32_t kS2BBytes = 4 * kS2SBO;   // 32 rows, one FP16 part
constexpr uint32_t kS2Stage = kS2ABytes + 2 * kS2BBytes;
constexpr uint32_t kS2Cols = 32;           // tensor-memory columns of a CTA
constexpr uint32_t kS2StgOff = 2 * kS2Stage;
constexpr uint32_t kS2RecOff = kS2StgOff + 32 * 64 * 4;
constexpr int kS2PerSm = 5;                // CTAs per SM: registers, shared memory; 160 tensor-memory columns
constexpr uint32_t kS2Smem = kS2RecOff + kSubItem * (8 + 8 + 4);

template <int W, int WIN>
__global__ void __launch_bounds__(kS2Threads, kS2PerSm) k_spread2_sub(const float2* __restrict__ f, float2* __restrict__ g, Geom geo,
                                                               Tiling tl, Bins bins) {
  static_assert(kI2Sub + W - 1 <= 31, "a sub-tile's window rows and columns must fit 32");
  static_assert(kSubItem <= kS2Threads, "one thread per node");
  constexpr int SH = off_bits(2);
  constexpr uint32_t MASK = (1u << SH) - 1u;
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ __align__(8) uint64_t bars[2];
  __shared__ uint32_t s_tmem;
  __shared__ float s_max[kS2Threads / 32];
  float* const stg = reinterpret_cast<float*>(smem + kS2StgOff);       // [32][64]
  float2* const rval = reinterpret_cast<float2*>(smem + kS2RecOff);    // [128] samples
  float2* const rfr = rval + kSubItem;                                 // [128] fractions
  uint32_t* const roff = reinterpret_cast<uint32_t*>(rfr + kSubItem);  // [128] o0 | o1 << 16
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int num = *bins.num_iitems, G = (int)gridDim.x;
  if (tid == 0) {
    tc::mbar_init(&bars[0], 1);
    tc::mbar_init(&bars[1], 1);
    tc::mbar_fence_init();
  }
  if (warp == 0) {
    tc::tmem_alloc(&s_tmem, kS2Cols);
    tc::tmem_relinquish();
  }
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  const uint32_t tmem = s_tmem;
  const int q = tid & 15, g8 = tid >> 4;  // operand task: node pair, row modulo 8
  const uint32_t word = (uint32_t)(q >> 2) * kS2LBO + (uint32_t)g8 * 16u + (uint32_t)(q & 3) * 4u;
  const float mf = (float)geo.m, norm = (float)geo.norm;
  const TapK k0 = tap_k<WIN>(geo, 0), k1 = tap_k<WIN>(geo, 1);
  const float2* sfrac = reinterpret_cast<const float2*>(bins.sfrac);
  const int64_t n0 = geo.n[0], n1 = geo.n[1];
  constexpr int E1 = kI2Sub + W - 1;
  const int E0 = min(tl.T[0], kI2Sub) + W - 1;
  const bool bulk = n1 >= E1 && (reinterpret_cast<uintptr_t>(g) & 15u) == 0 && (geo.ntot & 1) == 0;
  const uint32_t idesc = tc::idesc_f16(128, 32);
  uint32_t nst[2] = {0, 0};  // commits so far, per stage
  uint32_t gch = 0;
  bool failed = false;

  // this thread's node of the item: sample index two items ahead, record one item ahead
  int4 cur = (int)blockIdx.x < num ? bins.iitems[blockIdx.x] : make_int4(0, 0, 0, 0);
  int4 nxt = (int)blockIdx.x + G < num ? bins.iitems[blockIdx.x + G] : make_int4(0, 0, 0, 0);
  uint32_t r_off = 0;
  float2 r_fr = make_float2(0.f, 0.f), r_val = r_fr;
  int idx = cur.y + tid < cur.z ? bins.sidx[cur.y + tid] : -1;
  if (idx >= 0) {
    r_off = (uint32_t)bins.soff[cur.y + tid];
    r_fr = sfrac[cur.y + tid];
    r_val = f[idx];
  }
  idx = nxt.y + tid < nxt.z ? bins.sidx[nxt.y + tid] : -1;

  for (int it = blockIdx.x; it < num; it += G) {
    const int n = cur.z - cur.y;
    const I2Sub u = i2_decode(geo, tl, cur.x);
    {
      // windows relative to the sub-tile; past the item's end no window reaches a row
      const bool on = tid < n;
      const uint32_t o0 = on ? (r_off & MASK) - (uint32_t)u.s0 : 64u, o1 = on ? ((r_off >> SH) & MASK) - (uint32_t)u.s1 : 64u;
      roff[tid] = o0 | (o1 << 16);
      rfr[tid] = r_fr;
      rval[tid] = on ? r_val : make_float2(0.f, 0.f);
      const float m = on ? fmaxf(fabsf(r_val.x), fabsf(r_val.y)) : 0.f;
      const uint32_t mm = __reduce_max_sync(0xffffffffu, __float_as_uint(m));
      if (lane == 0) s_max[warp] = __uint_as_float(mm);
      if (tid < 32) tc::bulk_wait_read();  // the previous item's staging rows have been read
    }
    __syncthreads();
    const int4 next = nxt;
    if (idx >= 0) {  // the next item's record
      r_off = (uint32_t)bins.soff[next.y + tid];
      r_fr = sfrac[next.y + tid];
      r_val = f[idx];
    }
    nxt = it + 2 * G < num ? bins.iitems[it + 2 * G] : make_int4(0, 0, 0, 0);
    idx = nxt.y + tid < nxt.z ? bins.sidx[nxt.y + tid] : -1;
    int e = 0;
    frexpf(fmaxf(fmaxf(s_max[0], s_max[1]), fmaxf(s_max[2], s_max[3])) * norm, &e);
    e = max(e, -112);  // the scale stays a finite FP32 number
    const float scale = ldexpf(1.f, kTcLogB - e), bscale = norm * scale, unscale = ldexpf(1.f, e - kTcLogB - 10);

    const int nch = (n + kS2Chunk - 1) / kS2Chunk;
    uint32_t st = 0;
    for (int ch = 0; ch < nch && !failed; ++ch, ++gch) {
      st = gch & 1u;
      bool ok = true;
      if (gch >= 2) ok = tc::mbar_wait_spin(&bars[st], (nst[st] - 1u) & 1u, kTcPolls, 8);
      unsigned char* const sa = smem + st * kS2Stage;
      if (ok) {
        const int j = ch * kS2Chunk + 2 * q;
        const uint2 of = *reinterpret_cast<const uint2*>(roff + j);
        const float4 fr = *reinterpret_cast<const float4*>(rfr + j), val = *reinterpret_cast<const float4*>(rval + j);
        const int a0 = (int)(of.x & 0xffffu), a1 = (int)(of.x >> 16), b0 = (int)(of.y & 0xffffu), b1 = (int)(of.y >> 16);
        unsigned char* const sb = sa + kS2ABytes;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const int p = g8 + 8 * i;
          uint32_t hi, lo;
          tc_split2_f16(make_float2(tc_tap<WIN>(fr.x, mf, p - a0, W, k0) * kTcScaleA,
                                    tc_tap<WIN>(fr.z, mf, p - b0, W, k0) * kTcScaleA), hi, lo);
          *reinterpret_cast<uint32_t*>(sb + i * kS2SBO + word) = hi;
          *reinterpret_cast<uint32_t*>(sb + kS2BBytes + i * kS2SBO + word) = lo;
          const float wa = tc_tap<WIN>(fr.y, mf, p - a1, W, k1) * bscale, wb = tc_tap<WIN>(fr.w, mf, p - b1, W, k1) * bscale;
          tc_split2_f16(make_float2(wa * val.x, wb * val.z), hi, lo);
          *reinterpret_cast<uint32_t*>(sa + i * kS2SBO + word) = hi;
          *reinterpret_cast<uint32_t*>(sa + (8 + i) * kS2SBO + word) = lo;
          tc_split2_f16(make_float2(wa * val.y, wb * val.w), hi, lo);
          *reinterpret_cast<uint32_t*>(sa + (4 + i) * kS2SBO + word) = hi;
          *reinterpret_cast<uint32_t*>(sa + (12 + i) * kS2SBO + word) = lo;
        }
        tc::fence_proxy_async_smem();
      }
      failed = __syncthreads_or(!ok) != 0;
      if (tid == 0 && !failed) {
        tc::fence_after_sync();
        const uint32_t s0 = tc::smem_u32(sa);
        const uint64_t da = tc::smem_desc(s0, kS2LBO, kS2SBO), dh = tc::smem_desc(s0 + kS2ABytes, kS2LBO, kS2SBO),
                       dl = tc::smem_desc(s0 + kS2ABytes + kS2BBytes, kS2LBO, kS2SBO);
        const int ks = (min(kS2Chunk, n - ch * kS2Chunk) + 15) / 16;
        for (int k = 0; k < ks; ++k) {
          const uint64_t step = (uint64_t)(k * 2 * kS2LBO) >> 4;
          tc::mma_f16(tmem, da + step, dh + step, idesc, ch + k > 0 ? 1u : 0u);
          tc::mma_f16(tmem, da + step, dl + step, idesc, 1u);
        }
        tc::mma_commit(&bars[st]);
      }
      ++nst[st];
    }
    if (failed) break;
    // the sums: lo half (warps 2, 3) through the staging rows to the hi half (warps 0, 1)
    const bool ok = tc::mbar_wait_spin(&bars[st], (nst[st] - 1u) & 1u, kTcPolls, 8);
    if (__syncthreads_or(!ok)) {
      failed = true;
      break;
    }
    tc::fence_after_sync();
    float va[16], vb[16];
    const uint32_t acc = tmem + ((uint32_t)(32 * warp) << 16);
    tc::tmem_ld16(acc, va);
    tc::tmem_ld16(acc + 16u, vb);
    tc::tmem_ld_wait();
    tc::fence_before_sync();
    float* const col = stg + 2 * lane + (warp & 1);  // column p1 = lane, component warp % 2
    if (warp >= 2) {
#pragma unroll
      for (int i = 0; i < 16; ++i) {
        col[64 * i] = va[i];
        col[64 * (16 + i)] = vb[i];
      }
    }
    __syncthreads();
    if (warp < 2) {
#pragma unroll
      for (int i = 0; i < 16; ++i) {
        col[64 * i] = (va[i] + col[64 * i]) * unscale;
        col[64 * (16 + i)] = (vb[i] + col[64 * (16 + i)]) * unscale;
      }
    }
    tc::fence_proxy_async_smem();
    __syncthreads();
    const int64_t c0 = u.o.a[1] + u.s1;  // first column: a multiple of 16
    float2* const gi = g + u.o.inst * geo.ntot;
    if (bulk) {
      if (tid < E0) {
        float2* const row = gi + wrap_up(u.o.a[0] + u.s0 + tid, n0) * n1;
        const uint32_t src = tc::smem_u32(stg + 64 * tid);
        const int kw = (int)(n1 - c0 < 64 ? n1 - c0 : 64), cc = E1 < kw ? E1 : kw;  // columns before the row end (even)
        tc::bulk_reduce_add_f32(row + c0, src, (uint32_t)((cc + 1) & ~1) * 8u);
        if (kw < E1) tc::bulk_reduce_add_f32(row, src + (uint32_t)kw * 8u, (uint32_t)((E1 - kw + 1) & ~1) * 8u);
        tc::bulk_commit();
      }
    } else {
      for (int i = tid; i < E0 * E1; i += kS2Threads) {
        const int p0 = i / E1, p1 = i - p0 * E1;
        const float2 v = *reinterpret_cast<const float2*>(stg + 64 * p0 + 2 * p1);
        if (v.x != 0.f || v.y != 0.f)
          atomicAdd(gi + wrap_up(u.o.a[0] + u.s0 + p0, n0) * n1 + wrap_up(c0 + p1, n1), v);
      }
      __syncthreads();  // read before the next item's sums are staged
    }
    cur = next;
  }
  if (tid < 32) tc::bulk_wait_all();
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  if (warp == 0) tc::tmem_dealloc(tmem, kS2Cols);
  if (failed && tid == 0) atomicExch(bins.status, 2);
}

}  // namespace cg
