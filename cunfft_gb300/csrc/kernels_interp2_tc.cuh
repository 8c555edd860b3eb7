// kernels_interp2_tc.cuh -- 2D FP32 interpolation on the tensor cores (tcgen05, FP16 hi/lo x 3),
// sub-tiles streamed by TMA.
//
// The reference's 2D forward gridding (kernelConvWithGauss_2d, FGG form
// src/cunfft_kernel.cu:667-712: every node sums its (2m+2)^2 window of the oversampled grid
// with the weights psi_0 psi_1), with the same window-start rule and taps.  The binning
// orders every tile's nodes by sub-tile of 16 x 16 window starts (Tiling::ns sub-bins), and
// a work item is up to kSubItem = 128 nodes of one sub-tile.  For such a batch,
//     f_j = norm sum_{r} w0_j[r - l0_j] H[j, r],
//     H[j, (re|im, r)] = sum_{k} w1_j[k - l1_j] G[r, k] (re|im)
// with r over the sub-tile's 16 + W - 1 <= 31 rows and k over its 16 + W - 1 <= 31 columns
// (l0, l1: the node's window start inside the sub-tile).  H is the product D = A B^T of
//     A[j, k]               = w1_j[k - l1_j]           (128 nodes x K = 32, FP16 hi + lo, x 2^10)
//     B[(re|im, r), k]      = Re|Im G[r, k]            (N = 64 rows: real parts 0..31, imaginary 32..63)
// and the three products hi*hi + hi*lo + lo*hi accumulate in FP32 in tensor memory, node j
// in lane j.  The thread of node j finishes the sum over its W rows from its own lane.
//
// The grid is first split (k_split_rows) into FP16 hi + lo parts of its real and imaginary
// parts, each an array over the periodically padded index range [0, n_t + W - 1) per
// dimension, every padded row scaled by its own power of two 2^(14 - e_r) (2^e_r above its
// largest |Re|, |Im|); the node threads fold the inverse row scales into their w0 weights.
// A sub-tile's B then is one TMA box (hi re, hi im, lo re, lo im; 32 halves x 32 rows each)
// straight into the 64-byte swizzled K-major layout the MMAs read.
//
// Warp roles: two loader warps issue the TMA loads and stage the
// row scales, four warps issue the MMAs, two A sets of four warps build A and two reducing
// sets of four warps sum the accumulators over each node's rows; every role takes the CTA's
// items in turn.  Item li uses slot li % kI2Ring of A, B and the accumulators, so no warp
// waits for an MMA round trip between its own two jobs: loaders and A sets run up to kI2Ring
// items ahead of the MMAs, the reducing sets behind them.  Node records are loaded one item
// ahead, item descriptors two (a loader: 32 and more).  Hand-offs are mbarriers; every wait
// is bounded, and a wait that gives up raises the CTA's abort flag and the plan's device
// status flag, after which every role leaves its loop at its next wait and the kernel drains
// (bounded), frees its tensor memory and returns.
//
// What bounds it: the time one item takes in the slowest role, an issue latency and not a
// throughput (64 instances of a 512 x 512 grid, 6.8 M nodes in 98831 items, W = 12).  One
// thread that decoded each item and issued four boxes took 1660 cycles per item; decoding in
// 32 lanes and one box for all four parts bring it to 800, two loaders halve that.  One
// MMA-issuing thread took 1400 (three waits, six MMAs, three commits), four take 350 each.
// Items that fill only some of the 128 rows start at the quarter after the last one's end, so
// the four schedulers share them.  Together 695 -> 303 us (with the split 742 -> 350); now
// the reducing warps are busy 84 % of the time.  Eight issuers, four loaders or three sets
// of either kind are slower (395, 303, 355 us): they share the same issue slots.
#pragma once

#include <cuda.h>
#include <cuda_fp16.h>

#include "kernels_interp_tc.cuh"
#include "kernels_spread_tc.cuh"

namespace cg {

constexpr int kI2Sub = 16;                    // sub-tile extent of window starts per dimension
constexpr int kI2K = 32;                      // K: a sub-tile's 16 + W - 1 <= 31 columns, padded (one 64-byte row)
constexpr int kI2Rows = 32;                   // B rows per part: a sub-tile's 16 + W - 1 <= 31 rows, padded
constexpr int kI2N = 2 * kI2Rows;             // MMA N: real parts 0..31, imaginary parts 32..63
constexpr int kI2Sets = 2;                    // A-building sets and reducing sets, each on alternate items
constexpr int kI2Loaders = 2;                 // TMA warps, each on every kI2Loaders-th item
constexpr int kI2Issuers = 4;                 // MMA-issuing warps, each on every kI2Issuers-th item
constexpr int kI2AWarp0 = kI2Loaders + kI2Issuers;  // warps 6-13: two A sets of four warps
constexpr int kI2RWarp0 = kI2AWarp0 + 4 * kI2Sets;  // warps 14-21: two reducing sets of four warps
constexpr int kI2Threads = (kI2RWarp0 + 4 * kI2Sets) * 32;
constexpr int kI2Ring = 8;                    // slots of A, of B, and accumulators of kI2N columns (512 in all)
constexpr int kI2ABufs = kI2Ring, kI2Stages = kI2Ring, kI2Acc = kI2Ring;
constexpr int kI2Scales = 2 * kI2Ring;        // row-scale slots (item li's are read until its accumulator is)
constexpr uint32_t kI2Part = kI2Rows * 64u;   // one B part (hi re, hi im, lo re, lo im): 32 rows x 64 bytes
constexpr uint32_t kI2Stage = 4u * kI2Part;   // one slot of B, one TMA box: B hi = parts 0-1, B lo = parts 2-3
constexpr uint32_t kI2Polls = 1u << 20;       // mbarrier polls (<= 1 us each) before giving up

// 2D, 2m+2 in [4, 16], inner tile extent >= 16 (16-column sub-tiles whose TMA boxes start on
// 32-byte boundaries) and a row length divisible by 8 (16-byte rows of the split arrays; the
// split's quads never straddle the row's wrap)
__host__ __device__ constexpr bool interp2_tc_ok(int d, int W, int T1, int64_t n1) {
  return d == 2 && W >= 4 && W <= 16 && T1 >= kI2Sub && n1 >= 8 && n1 % 8 == 0;
}

// Shared-memory layout (byte offsets from a 1024-byte aligned base; host and device agree).
struct I2Layout {
  uint32_t b_off;      // kI2Ring B slots of kI2Stage
  uint32_t a_off;      // kI2Ring A slots x (A hi, A lo)
  uint32_t rs_off;     // kI2Scales x 32 floats: the row scales of an item's B rows
  uint32_t bar_off;    // afull[8], bfull[8], empty[8], tfull[8], tempty[8]; tensor-memory base; abort flag
  uint32_t total;      // bytes past the aligned base
  uint32_t dyn;        // dynamic shared memory to request (alignment slack included)
};

__host__ __device__ constexpr I2Layout i2_layout() {
  return I2Layout{0u,
                  kI2Ring * kI2Stage,
                  kI2Ring * kI2Stage + (uint32_t)kI2Ring * 2u * kItAPart,
                  kI2Ring * kI2Stage + (uint32_t)kI2Ring * 2u * kItAPart + (uint32_t)kI2Scales * 128u,
                  kI2Ring * kI2Stage + (uint32_t)kI2Ring * 2u * kItAPart + (uint32_t)kI2Scales * 128u + 512u,
                  kI2Ring * kI2Stage + (uint32_t)kI2Ring * 2u * kItAPart + (uint32_t)kI2Scales * 128u + 512u + 1024u};
}

// The taps of a node whose window starts at column (row) l0 of the sub-tile, in pairs of
// columns k, k + 1 = (0, 1), (2, 3), ... : next() gives the pair at k and steps to the next.
// Packed FP32x2 arithmetic for the Gaussian's exponents, one ex2 each, times 2^s; zero outside
// [l0, l0 + W), from a bit mask of the 32 columns (l0 >= 32: no node, every tap zero).  The
// same values as tc_tap<kWinGauss> times 2^s up to the last bits of ex2.  The pair's offsets
// l0 - k are exact small integers, stepped in FP32 instead of converted for every tap.
template <int W, int WIN>
struct TapPairs {
  uint32_t mask;
  float2 c, nl;  // fr + m; l0 - k, l0 - k - 1
  float fr, mf;
  int l0;
  __device__ __forceinline__ TapPairs(float fr_, float mf_, int l0_) : fr(fr_), mf(mf_), l0(l0_) {
    mask = l0 < 32 ? ((1u << W) - 1u) << l0 : 0u;
    c = make_float2(fr + mf, fr + mf);
    nl = make_float2((float)l0, (float)(l0 - 1));
  }
  __device__ __forceinline__ float2 next(int k, TapK tk, float s, float scale) {
    if (WIN == kWinGauss) {
      const float2 y = __fadd2_rn(c, nl);
      const float2 e = __ffma2_rn(__fmul2_rn(y, y), make_float2(-tk.a, -tk.a), make_float2(s, s));
      nl = __fadd2_rn(nl, make_float2(-2.f, -2.f));
      return make_float2(mask & (1u << k) ? tap_exp2(e.x) : 0.f, mask & (2u << k) ? tap_exp2(e.y) : 0.f);
    }
    return make_float2(tc_tap<WIN>(fr, mf, k - l0, W, tk) * scale, tc_tap<WIN>(fr, mf, k + 1 - l0, W, tk) * scale);
  }
};

// Padded split rows of a 2D grid, in the 3D split layout with one row per plane: half
// [batch][4][P0][P2s] with P0 = n0 + W - 1 padded rows, P1 = 1, P2 = n1 + W - 1 padded
// columns and P2s its multiple of 8.  Row scales: float [batch][P0], the inverse
// 2^(e - 14) of each padded row.
__host__ __device__ inline ItSplit i2_split_dims(const Geom& g) {
  ItSplit s;
  s.P0 = g.n[0] + g.W - 1;
  s.P1 = 1;
  s.P2 = g.n[1] + g.W - 1;
  s.P2s = (s.P2 + 7) / 8 * 8;
  return s;
}

constexpr int kI2SplitThreads = 256;

// The grid's padded FP16 hi/lo rows in one pass: warp w takes padded rows (instance, i0)
// w, w + nwarps, ...: it reads grid row i0 mod n0 once for its largest |Re|, |Im| (a warp
// reduction) and again (from L1: a row is n1 complex values) to write the row's P2s / 4
// quads of FP16 hi + lo parts of the real and imaginary parts, scaled by the row's
// 2^(14 - e), and the row's inverse scale.  A quad never straddles the row's wrap
// (n1 % 8 == 0).
static __global__ void __launch_bounds__(kI2SplitThreads) k_split_rows(const float2* __restrict__ g,
                                                                 __half* __restrict__ out,
                                                                 float* __restrict__ inv_scale, Geom geo, ItSplit sd) {
  const int lane = threadIdx.x & 31;
  const int64_t nwarps = ((int64_t)gridDim.x * blockDim.x) >> 5;
  const int64_t n0 = geo.n[0], n1 = geo.n[1], q4 = sd.P2s / 4, comp = sd.P0 * sd.P2s;
  const bool al16 = (reinterpret_cast<uintptr_t>(g) & 15u) == 0;  // n1 is a multiple of 8
  for (int64_t r = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; r < sd.P0 * geo.batch; r += nwarps) {
    const int64_t inst = r / sd.P0, i0 = r - inst * sd.P0;
    const float2* src = g + (inst * n0 + wrap_up(i0, n0)) * n1;
    float mx = 0.f;
    for (int64_t e = lane; e < n1 / 4; e += 32) {
      float4 a, b;
      ld_quad(src + 4 * e, al16, a, b);
      mx = fmaxf(mx, fmaxf(fmaxf(fmaxf(fabsf(a.x), fabsf(a.y)), fmaxf(fabsf(a.z), fabsf(a.w))),
                           fmaxf(fmaxf(fabsf(b.x), fabsf(b.y)), fmaxf(fabsf(b.z), fabsf(b.w)))));
    }
    const uint32_t m = __reduce_max_sync(0xffffffffu, __float_as_uint(mx));
    const int ex = it_plane_exp(__uint_as_float(m));
    const float scale = ldexpf(1.f, kItLogB - ex);
    if (lane == 0) inv_scale[inst * sd.P0 + i0] = ldexpf(1.f, ex - kItLogB);
    __half* const o_row = out + inst * 4 * comp + i0 * sd.P2s;
    for (int64_t e = lane; e < q4; e += 32) {
      const int64_t i1 = 4 * e;
      float4 a, b;
      ld_quad(src + wrap_up(i1, n1), al16, a, b);
      __half* o = o_row + i1;
      uint2 h, l;
      it_split4_f16(make_float4(a.x * scale, a.z * scale, b.x * scale, b.z * scale), h, l);
      *reinterpret_cast<uint2*>(o) = h;
      *reinterpret_cast<uint2*>(o + 2 * comp) = l;
      it_split4_f16(make_float4(a.y * scale, a.w * scale, b.y * scale, b.w * scale), h, l);
      *reinterpret_cast<uint2*>(o + comp) = h;
      *reinterpret_cast<uint2*>(o + 3 * comp) = l;
    }
  }
}

// An item's sub-tile inside its tile: sub-bin numbers and tiles' sub-bin counts are powers of two.
__device__ __forceinline__ int i2_sub_row(const Tiling& tl, int key) {
  return ((key & (tl.ns - 1)) >> (31 - __clz(tl.snb1))) << tl.ssh[0];
}
__device__ __forceinline__ int i2_sub_col(const Tiling& tl, int key) { return (key & (tl.snb1 - 1)) << tl.ssh[1]; }

// Sub-tile of an item: its tile's origin and instance, the sub-tile's offsets inside the tile
// (rows, columns), and its first row and column in the grid (tile origin + offset).
struct I2Sub {
  TileOrigin o;
  int r0, c0;
  int s0, s1;
};
__device__ __forceinline__ I2Sub i2_decode(const Geom& geo, const Tiling& tl, int key) {
  I2Sub u;
  u.o = decode_tile<2>(geo, tl, key >> (31 - __clz(tl.ns)));
  u.s0 = i2_sub_row(tl, key);
  u.s1 = i2_sub_col(tl, key);
  u.r0 = (int)u.o.a[0] + u.s0;
  u.c0 = (int)u.o.a[1] + u.s1;
  return u;
}

// Which 32 nodes of its set's next item a lane quarter takes, after an item of n nodes: the
// items' occupied quarters follow one another around the four lane quarters, so that the
// SM's four schedulers get the same share of items that fill only a part of the 128 rows.
__device__ __forceinline__ int i2_next_group(int ng, int n) { return (ng - ((n + 31) >> 5)) & 3; }

template <int W, int WIN>
__global__ void __launch_bounds__(kI2Threads, 1) k_interp2_tc(const __grid_constant__ CUtensorMap tmap,
                                                              const float* __restrict__ row_inv,
                                                              float2* __restrict__ f, Geom geo, Tiling tl, Bins bins) {
  constexpr int SH = off_bits(2);
  constexpr uint32_t MASK = (1u << SH) - 1u;
  static_assert(kI2Sub + W - 1 <= kI2K, "a sub-tile's columns must fit K");
  static_assert(kI2Sub + W - 1 <= kI2Rows, "a sub-tile's rows must fit one B part");
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  unsigned char* smem = smem_raw + ((1024u - (tc::smem_u32(smem_raw) & 1023u)) & 1023u);
  const I2Layout L = i2_layout();
  uint64_t* afull = reinterpret_cast<uint64_t*>(smem + L.bar_off);  // [8] A of the item built
  uint64_t* bfull = afull + kI2Ring;                                // [8] sub-tile landed (TMA)
  uint64_t* empty = bfull + kI2Ring;                                // [8] MMAs of the slot complete
  uint64_t* tfull = empty + kI2Ring;                                // [8] accumulator complete
  uint64_t* tempty = tfull + kI2Ring;                               // [8] accumulator read out
  float* const rsm = reinterpret_cast<float*>(smem + L.rs_off);
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(tempty + kI2Ring);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int num_items = *bins.num_iitems;
  const int G = (int)gridDim.x;
  // B rows of a sub-tile: the windows of 16 rows of window starts (16 + W - 1 <= 31); a
  // sub-tile of fewer rows (tiles of fewer than 16 rows) loads real grid rows past its own,
  // so that every B row the reduction weights is finite
  constexpr int kRows = kI2Sub + W - 1;

  if (tid == 0) {
    for (int i = 0; i < kI2Ring; ++i) {
      tc::mbar_init(&afull[i], 4);   // one arrival per warp of the A set
      tc::mbar_init(&bfull[i], 1);   // the loader's arrival (+ the box's bytes)
      tc::mbar_init(&empty[i], 1);
      tc::mbar_init(&tfull[i], 2);   // the MMAs' completion and the issuing thread's own arrival
      tc::mbar_init(&tempty[i], 4);  // one arrival per warp of the reducing set
    }
    *abort_flag = 0;
    tc::mbar_fence_init();
  }
  if (warp == 0) {
    tc::tmem_alloc(tmem_slot, 512);
    tc::tmem_relinquish();
  }
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  const uint32_t tmem = *tmem_slot;
  bool healthy = true;

  // Item li of this CTA (li = 0, 1, ...) is bins.iitems[blockIdx.x + li G]; it uses slot
  // li % kI2Ring of every ring in its cycle li / kI2Ring, and A set and reducing set
  // li % kI2Sets.
  if (warp < kI2Loaders) {
    // ======================= TMA: sub-tiles; their row scales =======================
    // The lanes decode 32 items at a time, one window ahead of their use.  Lane r loads the next item's row scale r and stores the current one's.
    const int64_t P0 = i2_split_dims(geo).P0;
    const int ld = warp;
    auto load_key = [&](uint32_t first) {  // this warp's items first, first + 1, ...
      const int64_t i = (int64_t)blockIdx.x + ((int64_t)(first + lane) * kI2Loaders + ld) * G;
      return i < num_items ? bins.iitems[i].x : 0;
    };
    auto row_scale = [&](int r0, int inst) {  // rows past the padded range: 0
      return lane < kRows && r0 + lane < P0 ? __ldg(row_inv + (int64_t)inst * P0 + r0 + lane) : 0.f;
    };
    struct Box {
      int r0, c0, inst;
    };
    auto decode = [&](int key) {
      const I2Sub u = i2_decode(geo, tl, key);
      return Box{u.r0, u.c0, (int)u.o.inst};
    };
    Box cur = decode(load_key(0)), next = cur;
    int key = load_key(32);
    float rs = row_scale(__shfl_sync(0xffffffffu, cur.r0, 0), __shfl_sync(0xffffffffu, cur.inst, 0));
    uint32_t li = (uint32_t)ld;
    for (int it = blockIdx.x + ld * G; it < num_items; it += kI2Loaders * G, li += kI2Loaders) {
      const uint32_t own = li / kI2Loaders;
      const int j = (int)(own & 31u), jn = (j + 1) & 31;
      if (j == 0) {
        if (own > 0) cur = next;
        next = decode(key);
        key = load_key(own + 64);
      }
      const int r0 = __shfl_sync(0xffffffffu, cur.r0, j), c0 = __shfl_sync(0xffffffffu, cur.c0, j);
      const int inst = __shfl_sync(0xffffffffu, cur.inst, j);
      const float rs_now = rs;
      const int r0n = __shfl_sync(0xffffffffu, jn ? cur.r0 : next.r0, jn);
      const int instn = __shfl_sync(0xffffffffu, jn ? cur.inst : next.inst, jn);
      if (it + kI2Loaders * G < num_items) rs = row_scale(r0n, instn);
      const uint32_t st = li % kI2Ring;
      const bool ok = li < (uint32_t)kI2Ring || tc::mbar_wait_warp(&empty[st], ((li / kI2Ring) - 1u) & 1u, kI2Polls);
      if (__any_sync(0xffffffffu, !ok || *abort_flag != 0)) {
        healthy = false;
        break;
      }
      // the MMAs of item li - 8 are complete, so the accumulator of item li - 16 was read out,
      // and with it the row-scale slot
      rsm[(li % kI2Scales) * 32 + lane] = rs_now;
      __syncwarp();
      if (lane == 0) {
        tc::mbar_arrive_expect_tx(&bfull[st], kI2Stage);
        // x = c0 is a multiple of 16 halves (tile and sub-tile origins): 32-byte aligned
        tc::tma_load_5d(smem + L.b_off + st * kI2Stage, &tmap, c0, r0, 0, 0, inst, &bfull[st]);
      }
    }
    // the boxes in flight have landed before this CTA can exit
    if (lane == 0)
      for (uint32_t k = kI2Loaders; k <= (uint32_t)kI2Ring && k <= li; k += kI2Loaders)
        healthy &= tc::mbar_wait_bounded(&bfull[(li - k) % kI2Ring], ((li - k) / kI2Ring) & 1u, kI2Polls);
    if (!healthy) *abort_flag = 1;
    __syncwarp();
  } else if (warp < kI2AWarp0) {
    // ======================= MMA issuers: lane 0 =======================
    if (lane == 0) {
      const uint32_t sa = tc::smem_u32(smem + L.a_off), sb = tc::smem_u32(smem + L.b_off);
      const uint32_t idesc = tc::idesc_f16(128, kI2N);
      uint32_t li = (uint32_t)(warp - kI2Loaders);
      for (int it = blockIdx.x + (warp - kI2Loaders) * G; it < num_items; it += kI2Issuers * G, li += kI2Issuers) {
        const uint32_t st = li % kI2Ring;
        bool ok = tc::mbar_wait_bounded(&afull[st], (li / kI2Ring) & 1u, kI2Polls);
        ok = ok && tc::mbar_wait_bounded(&bfull[st], (li / kI2Ring) & 1u, kI2Polls);
        if (ok && li >= (uint32_t)kI2Ring) ok = tc::mbar_wait_bounded(&tempty[st], ((li / kI2Ring) - 1u) & 1u, kI2Polls);
        if (!ok || *abort_flag != 0) {
          healthy = false;
          break;
        }
        tc::fence_after_sync();
        const uint32_t d = tmem + st * (uint32_t)kI2N;
        const uint64_t d_ah = tc::smem_desc(sa + st * 2u * kItAPart, kItLBO, kItSBOA);
        const uint64_t d_al = tc::smem_desc(sa + st * 2u * kItAPart + kItAPart, kItLBO, kItSBOA);
        const uint64_t d_bh = tc::smem_desc_sw64(sb + st * kI2Stage);
        const uint64_t d_bl = tc::smem_desc_sw64(sb + st * kI2Stage + 2u * kI2Part);
#pragma unroll
        for (int ks = 0; ks < kI2K / 16; ++ks) {
          const uint64_t ka = (uint64_t)((ks * 2 * kItLBO) >> 4);  // A: two core matrices per k-step
          const uint64_t kb = (uint64_t)((ks * 32) >> 4);          // B: 32 bytes into the swizzled row
          tc::mma_f16(d, d_ah + ka, d_bh + kb, idesc, ks > 0 ? 1u : 0u);
          tc::mma_f16(d, d_ah + ka, d_bl + kb, idesc, 1u);
          tc::mma_f16(d, d_al + ka, d_bh + kb, idesc, 1u);
        }
        tc::mma_commit(&empty[st]);
        tc::mma_commit(&tfull[st]);
        tc::mbar_arrive(&tfull[st]);  // hands the loader's row scales on to the reducing warps
      }
      // the last commits of each of this thread's slots: no arrival may land after exit (the
      // commits of one item complete together, so its empty covers its tfull)
      for (uint32_t k = kI2Issuers; k <= (uint32_t)kI2Ring && k <= li; k += kI2Issuers)
        healthy &= tc::mbar_wait_bounded(&empty[(li - k) % kI2Ring], ((li - k) / kI2Ring) & 1u, kI2Polls);
      if (!healthy) *abort_flag = 1;
    }
    __syncwarp();
  } else if (warp < kI2RWarp0) {
    // ======================= A sets: w1 over the sub-tile's 32 columns =======================
    // Set `set` takes the CTA's items set, set + 2, ...; warp (lane quarter q) builds the A
    // rows of nodes 32 q .. 32 q + 31 (slot = A row).  A quarter past the item's last node
    // skips its arithmetic but takes part in every hand-off.
    const int set = (warp - kI2AWarp0) >> 2, q = warp & 3, row = 32 * q + lane;
    const float mf = (float)geo.m;
    const TapK k1 = tap_k<WIN>(geo, 1);
    const float* sfrac = reinterpret_cast<const float*>(bins.sfrac);
    uint32_t li = (uint32_t)set;
    int it = blockIdx.x + set * G;
    // records of the next item, loaded one item ahead
    int4 nitem = it < num_items ? bins.iitems[it] : make_int4(0, 0, 1, 0);
    int4 fitem = it + kI2Sets * G < num_items ? bins.iitems[it + kI2Sets * G] : nitem;  // the item after it
    uint32_t noff = 0;
    float nfr = 0.f;
    int ng = q;  // the warp's node group in the next item
    if (it < num_items && 32 * ng + lane < nitem.z - nitem.y) {
      noff = (uint32_t)bins.soff[nitem.y + 32 * ng + lane];
      nfr = sfrac[(int64_t)(nitem.y + 32 * ng + lane) * 2 + 1];
    }
    for (; it < num_items; it += kI2Sets * G, li += kI2Sets) {
      const int4 cur = nitem;
      const uint32_t off = noff;
      const float fr1 = nfr;
      const int n = cur.z - cur.y, slot = 32 * ng + lane;
      const bool on = n > 32 * ng;  // warp-uniform
      const int itn = it + kI2Sets * G;
      ng = i2_next_group(ng, n);
      if (itn < num_items) {
        nitem = fitem;
        if (itn + kI2Sets * G < num_items) fitem = bins.iitems[itn + kI2Sets * G];
        if (32 * ng + lane < nitem.z - nitem.y) {
          noff = (uint32_t)bins.soff[nitem.y + 32 * ng + lane];
          nfr = sfrac[(int64_t)(nitem.y + 32 * ng + lane) * 2 + 1];
        }
      }
      const uint32_t ab = li % kI2Ring;
      if (li >= (uint32_t)kI2Ring) {  // the MMAs of item li - kI2Ring have read the slot
        const bool ok = tc::mbar_wait_warp(&empty[ab], ((li / kI2Ring) - 1u) & 1u, kI2Polls);
        if (__any_sync(0xffffffffu, !ok || *abort_flag != 0)) {  // the whole warp leaves together
          healthy = false;
          break;
        }
      } else if (__any_sync(0xffffffffu, *abort_flag != 0)) {
        healthy = false;
        break;
      }
      if (on) {
        const int s1 = i2_sub_col(tl, cur.x);
        const int l1 = slot < n ? (int)((off >> SH) & MASK) - s1 : 1 << 20;  // no node: every tap zero
        unsigned char* const ah = smem + L.a_off + ab * 2u * kItAPart;
        unsigned char* const al = ah + kItAPart;
        TapPairs<W, WIN> tp(fr1, mf, l1);
#pragma unroll
        for (int k8 = 0; k8 < kI2K / 8; ++k8) {
          uint32_t hi[4], lo[4];
#pragma unroll
          for (int v = 0; v < 4; ++v) {
            const int k = 8 * k8 + 2 * v;
            const float2 t = k < kI2Sub + W - 1 ? tp.next(k, k1, 10.f, kItScaleA)
                                                : make_float2(0.f, 0.f);
            tc_split2_f16(t, hi[v], lo[v]);
          }
          const uint32_t oa = (uint32_t)(row >> 3) * kItSBOA + (uint32_t)k8 * kItLBO + (uint32_t)(row & 7) * 16u;
          *reinterpret_cast<uint4*>(ah + oa) = make_uint4(hi[0], hi[1], hi[2], hi[3]);
          *reinterpret_cast<uint4*>(al + oa) = make_uint4(lo[0], lo[1], lo[2], lo[3]);
        }
      }
      tc::fence_proxy_async_smem();
      tc::mbar_arrive_warp(&afull[ab]);
    }
    if (!healthy) *abort_flag = 1;
  } else {
    // ======================= reducing sets: the accumulators =======================
    // Set `set` takes the CTA's items set, set + 2, ...; warp (lane quarter q) reduces TMEM
    // lanes 32 q .. 32 q + 31: node slot 32 q + lane sums its W rows of the accumulator with
    // its w0 weights and the rows' inverse scales.
    const int set = (warp - kI2RWarp0) >> 2, q = warp & 3;
    const float mf = (float)geo.m;
    const float norm = (float)geo.norm * (1.f / kItScaleA);
    const TapK k0 = tap_k<WIN>(geo, 0);
    const float* sfrac = reinterpret_cast<const float*>(bins.sfrac);
    uint32_t li = (uint32_t)set;
    int it = blockIdx.x + set * G;
    int4 nitem = it < num_items ? bins.iitems[it] : make_int4(0, 0, 1, 0);
    int4 fitem = it + kI2Sets * G < num_items ? bins.iitems[it + kI2Sets * G] : nitem;  // the item after it
    uint32_t noff = 0;
    float nfr = 0.f;
    int nidx = -1;
    int ng = q;
    if (it < num_items && 32 * ng + lane < nitem.z - nitem.y) {
      noff = (uint32_t)bins.soff[nitem.y + 32 * ng + lane];
      nfr = sfrac[(int64_t)(nitem.y + 32 * ng + lane) * 2];
      nidx = bins.sidx[nitem.y + 32 * ng + lane];
    }
    for (; it < num_items; it += kI2Sets * G, li += kI2Sets) {
      const int4 cur = nitem;
      const uint32_t off = noff;
      const float fr0 = nfr;
      const int idx = nidx;
      const int n = cur.z - cur.y, slot = 32 * ng + lane;
      const bool on = n > 32 * ng;  // warp-uniform
      const int itn = it + kI2Sets * G;
      ng = i2_next_group(ng, n);
      if (itn < num_items) {
        nitem = fitem;
        if (itn + kI2Sets * G < num_items) fitem = bins.iitems[itn + kI2Sets * G];
        nidx = -1;
        if (32 * ng + lane < nitem.z - nitem.y) {
          noff = (uint32_t)bins.soff[nitem.y + 32 * ng + lane];
          nfr = sfrac[(int64_t)(nitem.y + 32 * ng + lane) * 2];
          nidx = bins.sidx[nitem.y + 32 * ng + lane];
        }
      }
      const int l0 = slot < n ? (int)(off & MASK) - i2_sub_row(tl, cur.x) : 1 << 20;
      const float* const rs = rsm + (li % kI2Scales) * 32;  // the sub-tile's row scales
      const uint32_t acc = li % kI2Ring;
      const bool ok = tc::mbar_wait_warp(&tfull[acc], (li / kI2Ring) & 1u, kI2Polls);
      if (__any_sync(0xffffffffu, !ok || *abort_flag != 0)) {  // the whole warp leaves together
        healthy = false;
        break;
      }
      tc::fence_after_sync();
      float2 fs = make_float2(0.f, 0.f);
      if (on) {
        const uint32_t t0 = tmem + ((uint32_t)(32 * q) << 16) + acc * (uint32_t)kI2N;
        TapPairs<W, WIN> tp(fr0, mf, l0);
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          if (16 * h < kRows) {
            float vr[16], vi[16];
            tc::tmem_ld16(t0 + (uint32_t)(16 * h), vr);
            tc::tmem_ld16(t0 + (uint32_t)(kI2Rows + 16 * h), vi);
            tc::tmem_ld_wait();
#pragma unroll
            for (int c = 0; c < 16; c += 2) {
              const int r = 16 * h + c;
              if (r < kRows) {  // rows past kRows are never touched
                const float2 w = tp.next(r, k0, 0.f, 1.f);
                const float w0 = w.x * rs[r];
                fs.x = fmaf(w0, vr[c], fs.x);
                fs.y = fmaf(w0, vi[c], fs.y);
                if (r + 1 < kRows) {
                  const float w1 = w.y * rs[r + 1];
                  fs.x = fmaf(w1, vr[c + 1], fs.x);
                  fs.y = fmaf(w1, vi[c + 1], fs.y);
                }
              }
            }
          }
        }
      }
      tc::fence_before_sync();
      tc::mbar_arrive_warp(&tempty[acc]);
      if (idx >= 0) f[idx] = make_float2(fs.x * norm, fs.y * norm);
    }
    if (!healthy) *abort_flag = 1;
  }
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  if (warp == 0) tc::tmem_dealloc(tmem, 512);
  if (!healthy) atomicExch(bins.status, 2);
}

}  // namespace cg
