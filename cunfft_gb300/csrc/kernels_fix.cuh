// kernels_fix.cuh -- gridding of the FP64 form's transforms in 56-bit fixed point (fixmath.h).
//
// The bits below a tile's largest value are the same for all of its cells, and taps have an
// absolute error of 2^-54.  A transform's FFT mixes the cells anyway; the gridding stages alone,
// whose callers may look at single small cells, stay in FP64 (k_interp and k_spread of
// kernels_grid.cuh on the same tiles and items).
//
// Same method, work items and lane mapping as kernels_grid.cuh (the FP32 form's kernels);
// the arithmetic is integer because GB300's FP64 pipe (about 2 multiply-adds per clock and
// SM) bounds everything that goes through it, taps and reductions included.
//
//  * Interpolation: the staged tile is scaled by a power of two so that its largest
//    component is just below 2^vbits (55 for every usual window) and rounded to integers in
//    place; a node's sum is 6 integer multiply-adds per tap (complex value, real weight),
//    with the dimensions contracted one after the other.  Bound: the multiply-adds (29 per
//    clock and SM), then shared memory (16 bytes per tap).
//  * Spreading: an item's samples are scaled by their largest component, with headroom for
//    the item's node count; taps add to 64-bit integers in the shared-memory tile, so a
//    cell's sum does not depend on the order of its nodes, and the tile goes to the grid as
//    FP64 bulk reductions.  Bound: the multiply-adds, shared memory (32 bytes per tap) close
//    behind.
//  * Taps (Gaussian): one integer exponential per tap from two integers per node and
//    dimension, within 2^-54 of the largest tap; ES: the exponent in FP64, the exponential
//    in integers.
//  * Wide windows in 3D, whose padded tile does not fit in shared memory: the tile goes
//    through it in slabs of planes (SLAB), interpolation adding each slab's part of a node.
//  * Items whose values are not finite, or so large or small that the scaled results might
//    leave FP64's normal range, are computed in FP64 through global memory (one thread per
//    node), as are the samples of an item with a fraction that is not finite.
//
// Measured against the FP64-pipe kernels before: 3D n = 128^3, M = 2^18, m = 6 interpolation
// 4.18 -> 0.96 ms, spreading 5.75 -> 1.57 ms; m = 12 (global-memory kernels before)
// 68.8 -> 6.0 and 43.2 -> 9.9 ms; 2D n = 1024^2, M = 2^18, m = 6 0.80 -> 0.16 and
// 1.00 -> 0.28 ms.  Relative l2 error of whole transforms against 64-bit sums with exact taps
// (before, from the recurrence taps): m = 6 3e-16 to 1.2e-15 (2e-15 to 1.5e-14); 3D, m = 12,
// where the grid's values cancel 24-fold in the window's sum and the roll-off raises the
// spreading's rounding as much, forward 4e-16 to 9.8e-15 (9e-15 to 4.3e-14), adjoint 3e-16 to
// 6.1e-14 (1.5e-14 to 7.0e-14).
#pragma once

#include "fixmath.h"
#include "kernels_grid.cuh"

namespace cg {

constexpr int kFixMaxSmem = 227 * 1024 - 64;  // less the static variables
constexpr int kFixExpLo = 100, kFixExpHi = 1900;  // biased exponents the fixed-point path takes

// Warps and nodes per warp and round (interpolation), warps and nodes per batch (spreading).
// d = 3: the tile takes nearly all of the shared memory, so these share what is left.
__host__ __device__ constexpr int fix_interp_warps(int d) { return d == 3 ? 16 : 8; }
__host__ __device__ constexpr int fix_nodes_per_warp(int d) { return d == 1 ? 32 : (d == 3 ? 2 : 8); }
__host__ __device__ constexpr int fix_spread_warps(int d) { return d == 3 ? 16 : (d == 2 ? 8 : 4); }
// d = 3 in slabs: 40 nodes between barriers where they leave room for kFixSlabPlanes planes
__host__ __device__ constexpr int fix_batch(int d, int W) { return d == 3 ? (W > 14 && W <= 26 ? 40 : 20) : 64; }
// CTAs per SM the registers are limited for: in 1D and 2D an item is a few short phases
// between barriers, which other CTAs fill (2D, m = 6, M = 2^18: spreading 252 -> 223 us,
// interpolation 149 -> 140 us)
__host__ __device__ constexpr int fix_ctas(int d, int W, bool spread) {
  return d == 3 || W > 16 ? 1 : (spread && d == 2 ? 3 : 4);
}
// 1D spreading: node groups per warp (two windows of W <= 16 taps side by side)
__host__ __device__ constexpr int fix_spread_groups(int W) { return W <= 16 ? 2 : 1; }
// d = 3 spreading in slabs: planes per slab, one for each pair of warps.  Full slabs and a
// short last one: 33 planes (W = 26) as 8 + 8 + 8 + 8 + 1 instead of five of 7, where two of the
// 16 warps idle.  With 40 nodes per batch: n = 128^3, M = 2^18 adjoint, W = 18 6.49 -> 6.06 ms,
// W = 20 7.05 -> 6.54, W = 26 11.12 -> 10.24, W = 32 (no change) 14.75.
constexpr int kFixSlabPlanes = 8;

// Shared memory beyond the tile.
__host__ __device__ constexpr size_t fix_extra_smem(int d, int W, bool spread) {
  const size_t tab = sizeof(uint64_t) * kFixExpTab;
  // interpolation, per warp: taps (a pair's P and Q lie in front of its taps until these
  // are known), node and window start
  if (!spread) return tab + (size_t)fix_interp_warps(d) * fix_nodes_per_warp(d) * (d * W * sizeof(int2) + 2 * sizeof(int));
  // spreading, per node: taps, (P, Q), sample, sample x last-dimension taps, window start
  return tab + (size_t)fix_batch(d, W) * (d * W * sizeof(int2) + d * sizeof(FixGauss) + sizeof(int4) +
                                       (d > 1 ? W * sizeof(int4) : 0) + sizeof(int));
}

// Tile copies of the spreading kernel: in 1D every group of W lanes owns one.
__host__ __device__ constexpr int fix_tile_copies(int d, int W, bool spread) {
  return spread && d == 1 ? fix_spread_warps(1) * fix_spread_groups(W) : 1;
}

// Shared memory of a launch that stages the whole padded tile of outer extent E0.
__host__ __device__ constexpr size_t fix_smem_bytes(int d, int W, int E0, bool spread) {
  const size_t cells = d == 1 ? (size_t)E0 : (size_t)E0 * (d == 2 ? fix_row_stride(2, W) : fix_plane_stride(3, W));
  return sizeof(double2) * cells * fix_tile_copies(d, W, spread) + fix_extra_smem(d, W, spread);
}

__device__ __forceinline__ FixPair as_pair(int2 v) {
  FixPair p;
  p.hi = v.x;
  p.lo = v.y;
  return p;
}

// (P, Q) of a node and dimension (Gaussian), or its fraction (ES)
__device__ __forceinline__ FixGauss fix_stage(const Geom& geo, const FixPar& fp, int t, double fr) {
  if (geo.window == kWinES) {
    FixGauss g;
    g.P = __double_as_longlong(fr);
    g.Q = 0;
    return g;
  }
  const uint64_t c = t == 0 ? fp.c60[0] : (t == 1 ? fp.c60[1] : fp.c60[2]);
  return fix_gauss(__double2ll_rn(fr * 2305843009213693952.0), c);  // 2^61
}

// A lane's tap of a node and dimension: k = m - l and, per dimension, k^2 c (Gaussian).
template <int D>
struct FixTapLane {
  int k;
  int64_t k2c[D];
  __device__ __forceinline__ FixTapLane(const Geom& geo, const FixPar& fp, int l) : k(geo.m - l) {
#pragma unroll
    for (int t = 0; t < D; ++t) k2c[t] = (int64_t)(k * k) * fp.c57[t];
  }
  // tap of dimension t in units of 2^-BITS
  template <int BITS>
  __device__ __forceinline__ int64_t at(const Geom& geo, const FixPar& fp, int t, FixGauss s, const uint64_t* tab) const {
    if (geo.window == kWinES) {
      const double b = t == 0 ? fp.es_b2[0] : (t == 1 ? fp.es_b2[1] : fp.es_b2[2]);
      const double y = __longlong_as_double(s.P) + (double)k, z = 1.0 - (y * y) * geo.es_ia2;
      const double e = z > 0.0 ? b * (1.0 - sqrt(z)) : 64.0;
      return e < 63.0 ? fix_exp2neg<BITS>((uint64_t)__double2ll_rn(e * 144115188075855872.0), tab) : 0;  // 2^57
    }
    return fix_gauss_tap<BITS>(s, k, D == 1 || t == 0 ? k2c[0] : (D == 2 || t == 1 ? k2c[D > 1 ? 1 : 0] : k2c[D - 1]), tab);
  }
};

// A warp's rows of a tile of `rows` rows, E1 per plane: row = warp, warp + NW, ...
template <int D, int NW>
struct FixRows {
  int p0, p1, d0, d1, E1;
  __device__ __forceinline__ FixRows(int warp, int E1_) : E1(E1_) {
    p0 = D == 3 ? warp / E1 : warp;
    p1 = D == 3 ? warp - p0 * E1 : 0;
    d0 = D == 3 ? NW / E1 : NW;
    d1 = D == 3 ? NW - d0 * E1 : 0;
  }
  __device__ __forceinline__ void next() {
    p0 += d0;
    p1 += d1;
    if (D == 3 && p1 >= E1) {
      p1 -= E1;
      ++p0;
    }
  }
  __device__ __forceinline__ int cell(int S, int PS) const { return D == 3 ? p0 * PS + p1 * S : p0 * S; }
  // first element of the grid row (window starts a0, a1; n1 the last but one size in 3D)
  __device__ __forceinline__ int64_t base(const Geom& geo, const TileOrigin& o, int p_lo) const {
    uint32_t i0 = (uint32_t)o.a[0] + (uint32_t)(p0 + p_lo);
    while (i0 >= (uint32_t)geo.n[0]) i0 -= (uint32_t)geo.n[0];
    if (D == 2) return (int64_t)i0 * geo.n[1];
    uint32_t i1 = (uint32_t)o.a[1] + (uint32_t)p1;
    while (i1 >= (uint32_t)geo.n[1]) i1 -= (uint32_t)geo.n[1];
    return ((int64_t)i0 * geo.n[1] + i1) * geo.n[2];
  }
};

// High words of a complex value without their signs: the larger one holds the larger
// component's exponent.
__device__ __forceinline__ uint32_t fix_hi(double2 v) {
  return max((uint32_t)__double2hiint(v.x) & 0x7FFFFFFFu, (uint32_t)__double2hiint(v.y) & 0x7FFFFFFFu);
}

// Largest high word of the CTA (`slot` zero before; valid after the call's barrier)
__device__ __forceinline__ uint32_t fix_block_max(uint32_t hi, uint32_t* slot) {
  hi = __reduce_max_sync(0xffffffffu, hi);
  if ((threadIdx.x & 31) == 0) atomicMax(slot, hi);
  __syncthreads();
  return *slot;
}

// An item in FP64 through global memory, one thread per node.
template <int D, bool SPREAD>
__device__ __noinline__ void fix_item_f64(const double2* __restrict__ in, double2* __restrict__ out, const Geom& geo,
                                          const TileOrigin& o, const Bins& bins, const int4 item) {
  const double* sfrac = reinterpret_cast<const double*>(bins.sfrac);
  for (int64_t k = item.y + threadIdx.x; k < item.z; k += blockDim.x)
    grid_node_global<D, double, SPREAD>(in, out, geo, o, bins.sidx[k], (uint32_t)bins.soff[k], sfrac + k * D);
}

__device__ __forceinline__ int64_t shfl_xor_i64(int64_t v, int o) { return __shfl_xor_sync(0xffffffffu, v, o); }

// ---------------------------------------------------------------------------
// Interpolation
// ---------------------------------------------------------------------------
template <bool B>
struct BoolC {
  static constexpr bool value = B;
};

template <int D, int W, bool SLAB>
__global__ void __launch_bounds__(fix_interp_warps(D) * 32, fix_ctas(D, W, false))
    k_interp_fix(const double2* __restrict__ g, double2* __restrict__ f, Geom geo, Tiling tl, Bins bins, FixPar fp) {
  constexpr int R = kWarp / W, NIT = (W + R - 1) / R;
  constexpr bool FULL = R * NIT == W;
  constexpr int NB = fix_nodes_per_warp(D), NW = fix_interp_warps(D);
  constexpr int SH = off_bits(D);
  constexpr uint32_t MASK = (1u << SH) - 1u;
  constexpr int S = fix_row_stride(D, W), PS = fix_plane_stride(D, W);
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ int4 cur;
  __shared__ uint32_t s_key;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int tile_cells = D == 1 ? tl.E[0] : (D == 2 ? tl.E[0] * S : fp.planes * PS);
  int4* tile = reinterpret_cast<int4*>(smem);
  uint64_t* tab = reinterpret_cast<uint64_t*>(tile + tile_cells);
  int2* wb = reinterpret_cast<int2*>(tab + kFixExpTab) + warp * (NB * D * W);
  int* nrec = reinterpret_cast<int*>(reinterpret_cast<int2*>(tab + kFixExpTab) + NW * (NB * D * W)) + warp * 2 * NB;
  const int r = lane / W, l_last = lane - r * W;
  const bool lane_on = r < R;
  const double* sfrac = reinterpret_cast<const double*>(bins.sfrac);
  for (int i = threadIdx.x; i < kFixExpTab; i += blockDim.x) tab[i] = fix_exp_entry(i);
  const FixTapLane<D> taps(geo, fp, l_last);

  while (next_item(bins, 0, &cur)) {
    const int4 item = cur;
    const TileOrigin o = decode_tile<D>(geo, tl, item.x);
    const double2* gi = g + o.inst * geo.ntot;
    const int cnt = item.z - item.y;
    // nodes per warp and round: all warps busy on small items
    const int nbw = min(NB, (cnt + NW - 1) / NW);
    const int nslab = SLAB ? (tl.E[0] + fp.planes - 1) / fp.planes : 1;
    for (int sl = 0; sl < nslab; ++sl) {
      const int p_lo = SLAB ? sl * fp.planes : 0, p_n = SLAB ? min(fp.planes, tl.E[0] - p_lo) : tl.E[0];
      if (threadIdx.x == 0) s_key = 0;
      // stage the rows; every thread converts the elements it copied itself.  A lane's
      // columns are the same in every row.
      const int rows = D == 3 ? p_n * tl.E[1] : (D == 2 ? tl.E[0] : 1);
      const int e_last = tl.E[D - 1];
      constexpr int NC = D == 1 ? 1 : (fix_t_last(D) + W - 1 + kWarp - 1) / kWarp;
      double2* const td = reinterpret_cast<double2*>(tile);
      // fn(cell of the tile, row pointer of the grid, column of it) over this thread's elements
      auto each = [&](auto with_row, auto&& fn) {
        if constexpr (D == 1) {
          for (int p = threadIdx.x; p < e_last; p += NW * 32) fn(p, gi, wrap_up(o.a[0] + p, geo.n[0]));
        } else {
          int64_t col[NC];
#pragma unroll
          for (int c = 0; c < NC; ++c) col[c] = wrap_up(o.a[D - 1] + lane + c * kWarp, geo.n[D - 1]);
          FixRows<D, NW> rw(warp, tl.E[1]);
#pragma unroll 4
          for (int row = warp; row < rows; row += NW) {
            const double2* rp = gi;
            if (decltype(with_row)::value) rp += rw.base(geo, o, p_lo);
            const int dst = rw.cell(S, PS) + lane;
#pragma unroll
            for (int c = 0; c < NC; ++c)
              if (lane + c * kWarp < e_last) fn(dst + c * kWarp, rp, col[c]);
            rw.next();
          }
        }
      };
      each(BoolC<true>{}, [&](int d, const double2* rp, int64_t c) { cp_async_elem(td + d, rp + c); });
      cp_async_wait_all();
      uint32_t top = 0;
      each(BoolC<false>{}, [&](int d, const double2*, int64_t) { top = max(top, fix_hi(td[d])); });
      __syncthreads();  // s_key cleared
      top = fix_block_max(top, &s_key);
      const int key = fix_exp_of_hi(top);
      if (top != 0 && (key < kFixExpLo || key > kFixExpHi)) {
        fix_item_f64<D, false>(g, f, geo, o, bins, item);
        break;
      }
      const int sc = fp.vbits - (key - 1022);  // |v| 2^sc < 2^vbits
      each(BoolC<false>{}, [&](int d, const double2*, int64_t) {
        const double2 v = td[d];
        const FixPair x = fix_split(fix_from_f64(fix_bits(v.x), sc)), y = fix_split(fix_from_f64(fix_bits(v.y), sc));
        tile[d] = make_int4(x.hi, x.lo, y.hi, y.lo);
      });
      __syncthreads();

      int pf_idx = 0, pf_off = 0;  // records of the next batch, fetched one batch ahead
      double pf_fr = 0.0;
      auto fetch = [&](int at) {
        const int n = min(nbw, item.z - at);
        if (lane < n) {
          pf_idx = bins.sidx[at + lane];
          pf_off = bins.soff[at + lane];
        }
        if (lane < n * D) pf_fr = sfrac[(int64_t)at * D + lane];
      };
      fetch(item.y + warp * nbw);
      for (int bs = item.y + warp * nbw; bs < item.z; bs += NW * nbw) {
        const int nb = min(nbw, item.z - bs);
        bool bad = false;
        if (lane < nb) {
          nrec[lane] = pf_idx;
          nrec[NB + lane] = pf_off;
        }
        if (lane < nb * D) {
          bad = !(fabs(pf_fr) < 2.0);
          *reinterpret_cast<FixGauss*>(wb + lane * W) = fix_stage(geo, fp, lane % D, bad ? 0.0 : pf_fr);
        }
        const unsigned bads = __ballot_sync(0xffffffffu, bad);
        fetch(bs + NW * nbw);
        __syncwarp();
        for (int qt = r; qt - r < nb * D; qt += R) {
          const bool on = lane_on && qt < nb * D;
          FixPair w;
          if (on)
            w = fix_split_w(taps.template at<kFixOne>(geo, fp, qt % D, *reinterpret_cast<FixGauss*>(wb + qt * W), tab));
          __syncwarp();
          if (on) wb[qt * W + l_last] = make_int2(w.hi, w.lo);
        }
        __syncwarp();
        // value v of component (0: Re, 1: Im) of node q of the batch
        auto store = [&](int q, int comp, int64_t v) {
          const unsigned mine = (D == 1 ? 1u : (D == 2 ? 3u : 7u)) << (q * D);
          double* dst = reinterpret_cast<double*>(f + nrec[q]) + comp;
          double x = fix_to_f64(v, sc) * geo.norm;
          if (bads & mine) x = __longlong_as_double(0x7ff8000000000000ll);
          *dst = SLAB && sl > 0 ? *dst + x : x;
        };
        if constexpr (D == 1) {
          for (int q0 = 0; q0 < nb; q0 += R) {
            const int q = q0 + r;
            const bool on = lane_on && q < nb;
            FixSum sx, sy;
            if (on) {
              const int4 v = tile[((uint32_t)nrec[NB + q] & MASK) + l_last];
              const FixPair w = as_pair(wb[q * W + l_last]);
              fix_add(sx, as_pair(make_int2(v.x, v.y)), w);
              fix_add(sy, as_pair(make_int2(v.z, v.w)), w);
            }
            int64_t x = on ? fix_round(sx) : 0, y = on ? fix_round(sy) : 0;
#pragma unroll
            for (int s = 1; s < W; s <<= 1) {
              const int64_t x2 = __shfl_down_sync(0xffffffffu, x, s), y2 = __shfl_down_sync(0xffffffffu, y, s);
              if (l_last + s < W) {
                x += x2;
                y += y2;
              }
            }
            if (on && l_last == 0) {
              store(q, 0, x);
              store(q, 1, y);
            }
          }
        } else {
          // four nodes at a time: their lane sums are reduced together, each exchange
          // halving what a lane holds (nodes, then components)
          for (int q0 = 0; q0 < nb; q0 += 4) {
            int64_t ax[4], ay[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) {
              ax[u] = ay[u] = 0;
              const int q = q0 + u;
              if (q < nb && lane_on) {
                const uint32_t off = (uint32_t)nrec[NB + q];
                const int2* wq = wb + q * D * W;
                FixSum rx, ry;
                if constexpr (D == 3) {
                  const int o0 = off & MASK, o1 = (off >> SH) & MASK, o2 = off >> (2 * SH);
                  // planes of the window inside the slab
                  const int lo = SLAB ? max(0, p_lo - o0) : 0, hi = SLAB ? min(W, p_lo + p_n - o0) : W;
                  const int4* tb = tile + (o0 - p_lo) * PS + (o1 + r) * S + o2 + l_last;
                  if constexpr (SLAB) {
                    // planes outermost: their number varies, the rows are fixed
                    FixPair w1[NIT];
#pragma unroll
                    for (int it = 0; it < NIT; ++it) w1[it] = as_pair(wq[W + (FULL ? r + it * R : min(r + it * R, W - 1))]);
#pragma unroll 1
                    for (int l = lo; l < hi; ++l) {
                      FixSum px, py;
#pragma unroll
                      for (int it = 0; it < NIT; ++it) {
                        if (FULL || r + it * R < W) {
                          const int4 v = tb[l * PS + it * R * S];
                          fix_add(px, as_pair(make_int2(v.x, v.y)), w1[it]);
                          fix_add(py, as_pair(make_int2(v.z, v.w)), w1[it]);
                        }
                      }
                      const FixPair w0 = as_pair(wq[l]);
                      fix_add(rx, fix_split(fix_round(px)), w0);
                      fix_add(ry, fix_split(fix_round(py)), w0);
                    }
                  } else {
                    FixPair w0[W];
#pragma unroll
                    for (int l = 0; l < W; ++l) w0[l] = as_pair(wq[l]);
#pragma unroll
                    for (int it = 0; it < NIT; ++it) {
                      if (FULL || r + it * R < W) {
                        FixSum px, py;
#pragma unroll
                        for (int l = 0; l < W; ++l) {
                          const int4 v = tb[it * R * S + l * PS];
                          fix_add(px, as_pair(make_int2(v.x, v.y)), w0[l]);
                          fix_add(py, as_pair(make_int2(v.z, v.w)), w0[l]);
                        }
                        const FixPair w1 = as_pair(wq[W + r + it * R]);
                        fix_add(rx, fix_split(fix_round(px)), w1);
                        fix_add(ry, fix_split(fix_round(py)), w1);
                      }
                    }
                  }
                } else {
                  const int o0 = off & MASK, o1 = (off >> SH) & MASK;
                  const int4* tb = tile + (o0 + r) * S + o1 + l_last;
#pragma unroll
                  for (int it = 0; it < NIT; ++it) {
                    if (FULL || r + it * R < W) {
                      const int4 v = tb[it * R * S];
                      const FixPair w = as_pair(wq[r + it * R]);
                      fix_add(rx, as_pair(make_int2(v.x, v.y)), w);
                      fix_add(ry, as_pair(make_int2(v.z, v.w)), w);
                    }
                  }
                }
                const FixPair wl = as_pair(wq[(D - 1) * W + l_last]);
                ax[u] = fix_mul(fix_split(fix_round(rx)), wl);
                ay[u] = fix_mul(fix_split(fix_round(ry)), wl);
              }
            }
            __syncwarp();
            const bool h16 = lane & 16, h8 = lane & 8, h4 = lane & 4;
#pragma unroll
            for (int u = 0; u < 2; ++u) {
              const int64_t sx = h16 ? ax[u] : ax[u + 2], sy = h16 ? ay[u] : ay[u + 2];
              ax[u] = (h16 ? ax[u + 2] : ax[u]) + shfl_xor_i64(sx, 16);
              ay[u] = (h16 ? ay[u + 2] : ay[u]) + shfl_xor_i64(sy, 16);
            }
            const int64_t sx = h8 ? ax[0] : ax[1], sy = h8 ? ay[0] : ay[1];
            const int64_t x = (h8 ? ax[1] : ax[0]) + shfl_xor_i64(sx, 8), y = (h8 ? ay[1] : ay[0]) + shfl_xor_i64(sy, 8);
            int64_t v = (h4 ? y : x) + shfl_xor_i64(h4 ? x : y, 4);
            v += shfl_xor_i64(v, 2);
            v += shfl_xor_i64(v, 1);
            const int q = q0 + (h16 ? 2 : 0) + (h8 ? 1 : 0);
            if ((lane & 3) == 0 && q < nb) store(q, h4 ? 1 : 0, v);
          }
        }
        __syncwarp();
      }
      __syncthreads();
    }
    __syncthreads();  // the item is read by every thread before the next one is fetched
  }
}

// ---------------------------------------------------------------------------
// Spreading
// ---------------------------------------------------------------------------
__device__ __forceinline__ void bulk_add_f64(void* dst, uint32_t src, uint32_t bytes) {
  asm volatile("cp.reduce.async.bulk.global.shared::cta.bulk_group.add.f64 [%0], [%1], %2;" ::"l"(dst), "r"(src),
               "r"(bytes)
               : "memory");
}

// Adds (x, y) w to `n` <= G cells, i-th at cells[i * stride] with weight w[i * wstep].  Loads
// come before stores: the compiler cannot tell the cells from the weights behind them.
template <int G>
__device__ __forceinline__ void fix_cells_add(longlong2* cells, int stride, const int2* w, int wstep, int n, FixPair x,
                                              FixPair y) {
  longlong2 c[G];
  FixPair wi[G];
#pragma unroll
  for (int i = 0; i < G; ++i) {
    if (i < n) {
      wi[i] = as_pair(w[i * wstep]);
      c[i] = cells[i * stride];
    }
  }
#pragma unroll
  for (int i = 0; i < G; ++i) {
    c[i].x = fix_mad62(c[i].x, x, wi[i]);
    c[i].y = fix_mad62(c[i].y, y, wi[i]);
  }
#pragma unroll
  for (int i = 0; i < G; ++i)
    if (i < n) cells[i * stride] = c[i];
}

template <int D, int W, bool SLAB>
__global__ void __launch_bounds__(fix_spread_warps(D) * 32, fix_ctas(D, W, true))
    k_spread_fix(const double2* __restrict__ f, double2* __restrict__ g, Geom geo, Tiling tl, Bins bins, FixPar fp) {
  constexpr int R = kWarp / W;
  constexpr int NBC = fix_batch(D, W), NW = fix_spread_warps(D);
  constexpr int NP = D == 3 ? 2 : 1;  // d = 3: two warps share a row group, by plane parity
  constexpr int NG = NW / NP;
  constexpr int SH = off_bits(D);
  constexpr uint32_t MASK = (1u << SH) - 1u;
  constexpr int S = fix_row_stride(D, W), PS = fix_plane_stride(D, W);
  constexpr int COPIES = fix_tile_copies(D, W, true);
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ int4 cur;
  __shared__ uint32_t s_key;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int tile_cells = D == 1 ? tl.E[0] : (D == 2 ? tl.E[0] * S : fp.planes * PS);
  longlong2* tile = reinterpret_cast<longlong2*>(smem);
  int4* cval = reinterpret_cast<int4*>(tile + (size_t)tile_cells * COPIES);  // [NBC] samples
  int4* cv = cval + NBC;                                                    // [NBC][W] sample x last tap (d > 1)
  uint64_t* tab = reinterpret_cast<uint64_t*>(cv + (D > 1 ? NBC * W : 0));
  FixGauss* pq = reinterpret_cast<FixGauss*>(tab + kFixExpTab);
  int2* wb = reinterpret_cast<int2*>(pq + NBC * D);                          // [NBC][D][W]
  int* coff = reinterpret_cast<int*>(wb + NBC * D * W);                      // [NBC]
  const int r = lane / W, l_last = lane - r * W;
  const bool lane_on = r < R;
  const double* sfrac = reinterpret_cast<const double*>(bins.sfrac);
  for (int i = threadIdx.x; i < kFixExpTab; i += blockDim.x) tab[i] = fix_exp_entry(i);
  const FixTapLane<D> taps(geo, fp, l_last);

  while (next_item(bins, 1, &cur)) {
    const int4 item = cur;
    const TileOrigin o = decode_tile<D>(geo, tl, item.x);
    double2* gi = g + o.inst * geo.ntot;
    const int cnt = item.z - item.y;
    if (threadIdx.x == 0) s_key = 0;
    __syncthreads();
    uint32_t top = 0;
    for (int k = item.y + threadIdx.x; k < item.z; k += NW * 32) {
      const double2 v = f[bins.sidx[k]];
      top = max(top, fix_hi(make_double2(v.x * geo.norm, v.y * geo.norm)));
      for (int t = 0; t < D; ++t)
        if (!(fabs(sfrac[(int64_t)k * D + t]) < 2.0)) top = 0x7FFFFFFFu;
    }
    top = fix_block_max(top, &s_key);
    const int key = fix_exp_of_hi(top);
    if (top == 0) {  // all samples zero
      __syncthreads();
      continue;
    }
    if (key < kFixExpLo || key > kFixExpHi) {
      fix_item_f64<D, true>(f, g, geo, o, bins, item);
      __syncthreads();
      continue;
    }
    // a cell sums at most cnt samples times weights of at most one; each of the D products
    // takes two bits off the scale
    const int lc = cnt > 1 ? 32 - __clz(cnt - 1) : 0;
    const int sc = min(62, 62 + 2 * D - lc) - (key - 1022), sc_cell = sc - 2 * D;
    const int nslab = SLAB ? (tl.E[0] + fp.planes - 1) / fp.planes : 1;
    for (int sl = 0; sl < nslab; ++sl) {
      const int p_lo = SLAB ? sl * fp.planes : 0, p_n = SLAB ? min(fp.planes, tl.E[0] - p_lo) : tl.E[0];
      // records of a batch, fetched while the one before it runs: a fraction (thread = node and
      // dimension) and a sample with its window start (thread = node).  Adjoint of 64^3, M = 2^18:
      // m = 6 1.704 -> 1.671 ms, m = 8 6.10 -> 5.84, m = 12 10.16 -> 9.91
      static_assert(NBC * D <= NW * 32, "one record per thread");
      const int e = (int)threadIdx.x;
      double pf_fr = 0.0;
      double2 pf_v = make_double2(0.0, 0.0);
      int pf_off = 0;
      auto fetch = [&](int at) {
        const int n = min(NBC, item.z - at);
        if (e < n * D) pf_fr = sfrac[(int64_t)at * D + e];
        if (e < n) {
          pf_v = f[bins.sidx[at + e]];
          pf_off = bins.soff[at + e];
        }
      };
      fetch(item.y);
      for (int c = e; c < tile_cells * COPIES; c += NW * 32) tile[c] = make_longlong2(0, 0);
      for (int bs = item.y; bs < item.z; bs += NBC) {
        const int nb = min(NBC, item.z - bs);
        if (e < nb * D) pq[e] = fix_stage(geo, fp, e % D, pf_fr);
        if (e < nb) {
          const FixPair x = fix_split32(fix_from_f64(fix_bits(pf_v.x * geo.norm), sc)),
                        y = fix_split32(fix_from_f64(fix_bits(pf_v.y * geo.norm), sc));
          cval[e] = make_int4(x.hi, x.lo, y.hi, y.lo);
          coff[e] = pf_off;
        }
        fetch(bs + NBC);
        __syncthreads();
        for (int qt = warp * R + r; qt < nb * D && lane_on; qt += NW * R) {
          const int q = qt / D, t = qt - q * D;
          const FixPair w = fix_split32(taps.template at<62>(geo, fp, t, pq[qt], tab));
          wb[qt * W + l_last] = make_int2(w.hi, w.lo);
          if (D > 1 && t == D - 1) {  // the tap of the last dimension times the sample
            const int4 v = cval[q];
            const FixPair x = fix_split32(fix_mad62(0, as_pair(make_int2(v.x, v.y)), w)),
                          y = fix_split32(fix_mad62(0, as_pair(make_int2(v.z, v.w)), w));
            cv[q * W + l_last] = make_int4(x.hi, x.lo, y.hi, y.lo);
          }
        }
        __syncthreads();
        if constexpr (D == 1) {
          // lane group (warp, r) adds nodes warp * RG + r, + NW * RG, ... into its own copy;
          // a warp's lanes stay in step (a cell belongs to other lanes in the next node)
          constexpr int RG = fix_spread_groups(W);
          const bool mine = r < RG;
          longlong2* copy = tile + (size_t)(warp * RG + (mine ? r : 0)) * tile_cells;
          for (int q0 = warp * RG; q0 < nb; q0 += NW * RG) {
            const int q = q0 + r;
            if (mine && q < nb) {
              const int4 v = cval[q];
              fix_cells_add<1>(copy + ((uint32_t)coff[q] & MASK) + l_last, 0, wb + q * W + l_last, 0, 1,
                               as_pair(make_int2(v.x, v.y)), as_pair(make_int2(v.z, v.w)));
            }
            __syncwarp();
          }
        } else if constexpr (D == 2) {
          // warp w owns the row groups {g : g % NG == w}, group g = rows g R .. g R + R - 1
          // The products of four nodes are formed before their cells are touched.
          constexpr int U = 4, VIS = ((W + R - 2) / R + NG) / NG;  // visits: a window touches at most (W + R - 2) / R + 1 groups
          for (int q0 = 0; q0 < nb; q0 += U) {
#pragma unroll
            for (int vis = 0; vis < VIS; ++vis) {
              longlong2 pr[U];
              int cell[U];
#pragma unroll
              for (int u = 0; u < U; ++u) {
                const int q = min(q0 + u, nb - 1);
                const uint32_t off = (uint32_t)coff[q];
                const int o0 = off & MASK, o1 = (off >> SH) & MASK;
                const int g_first = o0 / R;
                const int row = (g_first + ((warp - g_first) & (NG - 1)) + vis * NG) * R + r, l0 = row - o0;
                const bool on = lane_on && l0 >= 0 && l0 < W && q0 + u < nb;
                const int4 v = cv[q * W + (lane_on ? l_last : 0)];
                const FixPair w = as_pair(wb[q * 2 * W + (on ? l0 : 0)]);
                pr[u].x = fix_mad62(0, as_pair(make_int2(v.x, v.y)), w);
                pr[u].y = fix_mad62(0, as_pair(make_int2(v.z, v.w)), w);
                cell[u] = on ? row * S + o1 + l_last : -1;
              }
#pragma unroll
              for (int u = 0; u < U; ++u) {
                if (cell[u] >= 0) {
                  longlong2 c = tile[cell[u]];
                  c.x += pr[u].x;
                  c.y += pr[u].y;
                  tile[cell[u]] = c;
                }
                __syncwarp();  // a cell belongs to other lanes in the next node
              }
            }
          }
        } else {
          const int wg = warp & (NG - 1), par = warp / NG;
          for (int q = 0; q < nb; ++q) {
            const uint32_t off = (uint32_t)coff[q];
            const int o0 = off & MASK, o1 = (off >> SH) & MASK, o2 = off >> (D == 3 ? 2 * SH : 0);
            const int2* wq = wb + q * 3 * W;
            const int4 v = cv[q * W + (lane_on ? l_last : 0)];
            const FixPair vx = as_pair(make_int2(v.x, v.y)), vy = as_pair(make_int2(v.z, v.w));
            if constexpr (SLAB) {
              // warp w owns plane w % NG of the slab, on the row groups of parity w / NG
              const int l0 = p_lo + wg - o0;
              if (wg < p_n && l0 >= 0 && l0 < W) {  // the same for the whole warp
                const FixPair w0 = as_pair(wq[l0]);
                const FixPair x = fix_split32(fix_mad62(0, vx, w0)), y = fix_split32(fix_mad62(0, vy, w0));
                longlong2* tb = tile + wg * PS + o2 + l_last;
                const int g_first = o1 / R, g0 = g_first + ((par - g_first) & 1);
                constexpr int C = ((W + R - 2) / R + 2) / 2, G = (C + (C + 6) / 7 - 1) / ((C + 6) / 7);
#pragma unroll
                for (int i = 0; i < C; i += G) {
                  const int row = (g0 + 2 * i) * R + r, l1 = row - o1;
                  // rows l1, l1 + 2 R, ... below W; a first row of l1 < 0 is skipped
                  const int n = lane_on && l1 < W ? min(min(G, C - i), (W - 1 - l1) / (2 * R) + 1) : 0;
                  const int skip = l1 < 0 ? 1 : 0;
                  fix_cells_add<G>(tb + (row + 2 * R * skip) * S, 2 * R * S, wq + W + l1 + 2 * R * skip, 2 * R, n - skip, x, y);
                }
              }
            } else {
              // warp w owns the row groups {g : g % NG == w % NG} on the planes of parity w / NG
              const int g_first = o1 / R, g_last = (o1 + W - 1) / R;
              for (int gg = g_first + ((wg - g_first) & (NG - 1)); gg <= g_last; gg += NG) {
                const int l1 = gg * R + r - o1;
                if (lane_on && l1 >= 0 && l1 < W) {
                  const FixPair w1 = as_pair(wq[W + l1]);
                  const FixPair x = fix_split32(fix_mad62(0, vx, w1)), y = fix_split32(fix_mad62(0, vy, w1));
                  longlong2* tb = tile + o0 * PS + (gg * R + r) * S + o2 + l_last;
                  const int l0 = (par - o0) & 1;
                  constexpr int C = W / NP, G = (C + (C + 6) / 7 - 1) / ((C + 6) / 7);  // groups of at most 7
#pragma unroll
                  for (int i = 0; i < C; i += G)
                    fix_cells_add<G>(tb + (l0 + NP * i) * PS, NP * PS, wq + l0 + NP * i, NP, min(G, C - i), x, y);
                }
              }
            }
            __syncwarp();  // a cell belongs to other lanes in the next node
          }
        }
        __syncthreads();
      }
      // integers to FP64 in place (d = 1: the copies folded into the first), then to the grid
      const int rows = D == 3 ? p_n * tl.E[1] : (D == 2 ? tl.E[0] : 1);
      const int e_last = tl.E[D - 1];
      const int64_t a_last = o.a[D - 1], n_last = geo.n[D - 1];
      double2* const dt = reinterpret_cast<double2*>(tile);
      const bool bulk = D > 1 && n_last >= e_last && (reinterpret_cast<uintptr_t>(gi) & 15u) == 0;
      if constexpr (D == 1) {
        for (int p = threadIdx.x; p < e_last; p += NW * 32) {
          longlong2 c = tile[p];
          for (int k = 1; k < COPIES; ++k) {
            const longlong2 b = tile[(size_t)k * tile_cells + p];
            c.x += b.x;
            c.y += b.y;
          }
          if (c.x | c.y)
            global_add(gi + wrap_up(a_last + p, n_last), make_double2(fix_to_f64(c.x, sc_cell), fix_to_f64(c.y, sc_cell)));
        }
      } else {
        const int c1 = (int)(n_last - a_last < e_last ? n_last - a_last : e_last);  // columns before the row end
        constexpr int NC = (fix_t_last(D) + W - 1 + kWarp - 1) / kWarp;
        FixRows<D, NW> rw(warp, tl.E[1]);
#pragma unroll 2
        for (int row = warp; row < rows; row += NW) {
          const int src = rw.cell(S, PS);
          double2* const gr = gi + rw.base(geo, o, p_lo);
          bool any = false;
#pragma unroll
          for (int c = 0; c < NC; ++c) {
            const int p = lane + c * kWarp;
            if (p < e_last) {
              const longlong2 b = tile[src + p];
              const double2 v = make_double2(fix_to_f64(b.x, sc_cell), fix_to_f64(b.y, sc_cell));
              const bool set = (b.x | b.y) != 0;
              any |= set;
              if (bulk) dt[src + p] = v;
              else if (set) global_add(gr + wrap_up(a_last + p, n_last), v);
            }
          }
          if (bulk && __any_sync(0xffffffffu, any)) {
            // one contiguous run, or two when the row wraps
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            __syncwarp();
            if (lane == 0) {
              const uint32_t s0 = (uint32_t)__cvta_generic_to_shared(dt + src);
              bulk_add_f64(gr + a_last, s0, (uint32_t)c1 * 16u);
              if (c1 < e_last) bulk_add_f64(gr, s0 + (uint32_t)c1 * 16u, (uint32_t)(e_last - c1) * 16u);
              asm volatile("cp.async.bulk.commit_group;" ::: "memory");
            }
          }
          rw.next();
        }
        // the copy engine has read the tile before it is cleared again
        if (lane == 0) asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
      }
      __syncthreads();
    }
  }
  if (D > 1 && lane == 0) asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
}

}  // namespace cg
