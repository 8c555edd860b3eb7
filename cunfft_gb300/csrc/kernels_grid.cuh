// kernels_grid.cuh -- tiled Gaussian gridding: interpolation (forward) and spreading (adjoint)
// of the FP32 form, and of the FP64 form's stages on their own (its transforms grid in
// kernels_fix.cuh).
//
// Method (the reference's, src/cunfft_kernel.cu:514-1149): node j touches the
// (2m+2)^d grid points (u_t + l_t) mod n_t, l_t = 0..2m+1, with weight
// prod_t psi_t(l_t), psi(l) = sqrt(b') exp(-(c - l)^2 / b), c = n x - u.
//
// GB300 design:
//  * Work items: a tile of the grid (T0 x T1 x T2 window starts) plus at most
//    `chunk` of its sorted nodes.  A persistent grid of CTAs pulls items from an
//    atomic queue, so clustered node sets (thousands of nodes in one tile) spread
//    over many CTAs instead of serialising on one.
//  * The CTA stages the padded tile (T_t + W - 1 per dim, wrapped mod n) in shared
//    memory.  The inner strides are compile-time constants (common.cuh): row
//    stride S == W (mod 16) elements, so the lane -> tap mapping below touches
//    consecutive banks (no conflicts for float2 or double2 elements), and every
//    tap offset is an immediate.
//  * Lane i < R*W (R = 32/W) owns innermost tap l_last = i % W and rows
//    r = i / W, r + R, ... of the remaining taps (for d = 3 a row is an (l0, l1)
//    pair walked over the 2m+2 planes l0).
//  * Interpolation: one warp per node at a time; the warp reduces the sums of four
//    nodes together with shuffles.  Node records and tap weights (a lane per tap) of a
//    batch of nodes are staged per warp in shared memory; the next batch's records
//    are fetched into registers while the current batch runs.  Bound: instruction
//    issue (staging, taps and reductions beside 2 instructions per lane and tap).  A
//    lane per tap instead of one per node and dimension, staging without divisions,
//    equal batches per warp and the joint reduction: 3D grid 110 x 84 x 126, W = 10,
//    1e5 nodes: forward + adjoint + binning 208 -> 180 us (this kernel 103 us before).
//  * Spreading: no shared-memory atomics (a float atomic add on shared memory is a
//    compare-and-swap loop).  Every warp walks all nodes of a CTA-wide batch but
//    writes only the planes (d = 3) or row groups (d = 2) it owns, with plain
//    load / FMA / store; for d = 1 each warp accumulates into a private copy of
//    the tile.  Batches are double-buffered (one barrier per batch).  The tile is
//    then added to the global grid with vector atomics, so neighbouring items'
//    halos combine.  In 1D and 2D eight CTAs form a cluster, take neighbouring items
//    and add the tiles of one grid tile over their shared memory first: shorter items
//    for the SMs (eight times as many partial sums on a cell, added in FP32) had raised
//    the error of dense grids of few tiles (N = 173, m = 4, M = 1e5: 2.1e-7 with items of
//    2048 nodes, 3.0e-7 with 256, 2.1e-7 with 256 in clusters; adjoint 113, 54, 58 us).
//  * Wide windows in 3D: above 16 taps a warp's lanes take consecutive cells of a plane's
//    W x W window (interpolation; one row of W taps per pass left 32 - W lanes idle), and
//    above 24 taps, where the padded tile of a single plane of window starts does not fit
//    in shared memory, the tile goes through it in slabs of planes, interpolation adding
//    each slab's part of a node.  n = 128^3, M = 2^18, interpolation with roll-off and FFT:
//    W = 18 1.45 -> 0.99 ms, W = 22 2.08 -> 1.46; W = 26 17.0 -> 2.24 and spreading 20.2 ->
//    4.54 (one thread per node through global memory before).
//  * Tap weights: one hardware exp2 per tap in the FP32 form; in the FP64 form the reference's
//    fast-Gaussian-gridding recurrence (src/cunfft_kernel.cu:491-505) from the middle tap
//    outwards (4 exp per node and dim), which keeps the scarce FP64 pipe on the taps.
#pragma once

#include "runtime.h"

namespace cg {

// Compile-time extents and strides of the staged tile of elements C, and whether windows of W
// taps go through it in slabs of planes.
template <int D, int W, typename C>
struct TileShape {
  static constexpr bool F64 = sizeof(C) == 16;
  static constexpr int S = F64 ? fix_row_stride(D, W) : fixed_row_stride(D, W);
  static constexpr int PS = F64 ? fix_plane_stride(D, W) : fixed_plane_stride(D, W);
  static constexpr int LAST = F64 ? fix_t_last(D) : fixed_t_last(D, W);
  static constexpr bool SLAB = F64 ? D == 3 && W > kFixWholeW : grid_slabs(D, W);
};

// bits of the packed tile-local window start, per dimension
__host__ __device__ constexpr int off_bits(int d) { return d == 1 ? 30 : (d == 2 ? 15 : 10); }

template <typename T> struct WeightMath;

template <> struct WeightMath<float> {
  // Gaussian: psi(l) / sqrt(b') = exp(-(fr + m - l)^2 / b) = exp2(-(y*y) * log2(e)/b);
  // ES: exp(beta (sqrt(1 - y^2/alpha^2) - 1)), y = fr + m - l
  static __device__ __forceinline__ float tap(float y, const Geom& g, int t) {
    const TapK k = tap_k(g, t);
    return g.window == kWinES ? win_tap<kWinES>(y, k) : win_tap<kWinGauss>(y, k);
  }
  static __device__ __forceinline__ void taps(float fr, int m, const Geom& g, int t, int W, float* out) {
    const TapK k = tap_k(g, t);
    if (g.window == kWinES) {
#pragma unroll 4
      for (int l = 0; l < W; ++l) out[l] = win_tap<kWinES>(fr + (float)(m - l), k);
    } else {
#pragma unroll 4
      for (int l = 0; l < W; ++l) out[l] = win_tap<kWinGauss>(fr + (float)(m - l), k);
    }
  }
};

template <> struct WeightMath<double> {
  // FGG form about the middle tap k = l - m = 0: psi_k = phi E^k exp(-k^2/b), phi = exp(-fr^2/b),
  // E = exp(2 fr/b).  From the first tap on (c = m + fr in place of fr) every tap had the relative
  // error of phi = exp(-c^2/b), some c^2/b = 20 roundings; here the large taps have a few.
  static __device__ __forceinline__ void taps(double fr, int m, const Geom& g, int t, int W, double* out) {
    if (g.window == kWinES) {  // exp(beta (sqrt(1 - y^2/alpha^2) - 1)), zero outside |y| < alpha
      const double beta = t == 0 ? g.es_beta[0] : (t == 1 ? g.es_beta[1] : g.es_beta[2]);
      const double c = (double)m + fr;
      for (int l = 0; l < W; ++l) {
        const double y = c - (double)l, z = 1.0 - (y * y) * g.es_ia2;
        out[l] = z > 0.0 ? exp(beta * (sqrt(z) - 1.0)) : 0.0;
      }
      return;
    }
    const double b = t == 0 ? g.b[0] : (t == 1 ? g.b[1] : g.b[2]);
    const double ib = 1.0 / b;
    const double E = exp(2.0 * fr * ib), Ei = exp(-2.0 * fr * ib);
    const double q = exp(-ib);  // exp(-k^2/b) by the recurrence of src/cunfft.cu:60-76
    double er = exp(-(fr * fr) * ib), el = er, gk = 1.0, qstep = q;  // phi E^k, phi E^-k, exp(-k^2/b), exp(-(2k+1)/b)
    out[m] = er;
#pragma unroll 4
    for (int k = 1; k <= m + 1; ++k) {
      er *= E;
      el *= Ei;
      gk *= qstep;
      qstep *= q * q;
      out[m + k] = er * gk;
      if (k <= m) out[m - k] = el * gk;
    }
  }
};

__device__ __forceinline__ float2 cmul_add(float2 acc, float w, float2 v) {
  return __ffma2_rn(make_float2(w, w), v, acc);
}
__device__ __forceinline__ double2 cmul_add(double2 acc, double w, double2 v) {
  acc.x = fma(w, v.x, acc.x);
  acc.y = fma(w, v.y, acc.y);
  return acc;
}
// A weight ready for the complex multiply-add: the (w, w) pair of a packed f32x2 FMA.
template <typename T> struct WPair;
template <> struct WPair<float> {
  using t = float2;
  static __device__ __forceinline__ float2 make(float w) { return make_float2(w, w); }
};
__device__ __forceinline__ float2 cmul_addp(float2 acc, float2 ww, float2 v) { return __ffma2_rn(ww, v, acc); }
template <> struct WPair<double> {
  using t = double;
  static __device__ __forceinline__ double make(double w) { return w; }
};
__device__ __forceinline__ double2 cmul_addp(double2 acc, double w, double2 v) { return cmul_add(acc, w, v); }

// Asynchronous global -> shared copy of one complex element (cp.async, 8 or 16 bytes).
template <typename C>
__device__ __forceinline__ void cp_async_elem(C* dst, const C* src) {
  const unsigned s = (unsigned)__cvta_generic_to_shared(dst);
  if constexpr (sizeof(C) == 16)
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(s), "l"(src) : "memory");
  else
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(s), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;\n" ::: "memory"); }

__device__ __forceinline__ float2 cscale(float2 v, float w) { return __fmul2_rn(make_float2(w, w), v); }
__device__ __forceinline__ double2 cscale(double2 v, double w) { return make_double2(v.x * w, v.y * w); }

__device__ __forceinline__ void global_add(float2* p, float2 v) { atomicAdd(p, v); }
__device__ __forceinline__ void global_add(double2* p, double2 v) {
  atomicAdd(&p->x, v.x);
  atomicAdd(&p->y, v.y);
}

template <typename C>
__device__ __forceinline__ C czero() {
  C z;
  z.x = 0;
  z.y = 0;
  return z;
}

template <typename C>
__device__ __forceinline__ C shfl_xor_c(C v, int o) {
  v.x = __shfl_xor_sync(0xffffffffu, v.x, o);
  v.y = __shfl_xor_sync(0xffffffffu, v.y, o);
  return v;
}

// Tile origin a_t of a work item's tile and its instance.
struct TileOrigin {
  int64_t inst;
  int64_t a[kMaxDim];
};

template <int D>
__device__ __forceinline__ TileOrigin decode_tile(const Geom& geo, const Tiling& tl, int64_t tile) {
  TileOrigin o;
  o.inst = tile / tl.tiles_per_inst;
  int64_t lt = tile - o.inst * tl.tiles_per_inst;
  o.a[0] = o.a[1] = o.a[2] = 0;
  if (D == 3) {
    o.a[2] = (lt % tl.nb[2]) * tl.T[2];
    lt /= tl.nb[2];
  }
  if (D >= 2) {
    o.a[1] = (lt % tl.nb[1]) * tl.T[1];
    lt /= tl.nb[1];
  }
  o.a[0] = lt * tl.T[0];
  return o;
}

// Rows of the staged tile: [E0][E1] for d = 3, [E0] for d = 2, one for d = 1.
// The shared-memory row of (p0, p1) starts at p0 * PS + p1 * S.
template <int D>
__device__ __forceinline__ int tile_rows(const Tiling& tl) {
  return D == 3 ? tl.E[0] * tl.E[1] : (D == 2 ? tl.E[0] : 1);
}

template <int D>
__device__ __forceinline__ void row_coords(const Tiling& tl, int row, int* p0, int* p1) {
  if (D == 3) {
    *p0 = row / tl.E[1];
    *p1 = row - *p0 * tl.E[1];
  } else {
    *p0 = row;
    *p1 = 0;
  }
}

template <int D>
__device__ __forceinline__ int64_t row_gbase(const Geom& geo, const TileOrigin& o, int p0, int p1) {
  if (D == 3) return (wrap_up(o.a[0] + p0, geo.n[0]) * geo.n[1] + wrap_up(o.a[1] + p1, geo.n[1])) * geo.n[2];
  if (D == 2) return wrap_up(o.a[0] + p0, geo.n[0]) * geo.n[1];
  return 0;
}

template <int D, int W, typename C>
__device__ __forceinline__ void load_tile(C* tile, const C* __restrict__ gi, const Geom& geo, const Tiling& tl,
                                          const TileOrigin& o, int p_lo, int p_n) {
  constexpr int S = TileShape<D, W, C>::S, PS = TileShape<D, W, C>::PS;
  const int E_last = tl.E[D - 1];
  const int64_t n_last = geo.n[D - 1], a_last = o.a[D - 1];
  if (D == 1) {
    for (int p = threadIdx.x; p < E_last; p += blockDim.x) cp_async_elem(tile + p, gi + wrap_up(a_last + p, n_last));
    cp_async_wait_all();
    return;
  }
  // A lane's columns are the same in every row, and a warp steps from row to row without
  // divisions: the staging was a third of the instructions of an item of some 80 nodes.
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
  const int rows = D == 3 ? p_n * tl.E[1] : tile_rows<D>(tl), E1 = tl.E[1];
  constexpr int NC = (TileShape<D, W, C>::LAST + W - 1 + kWarp - 1) / kWarp;
  int64_t col[NC];
#pragma unroll
  for (int c = 0; c < NC; ++c) col[c] = lane + c * kWarp < E_last ? wrap_up(a_last + lane + c * kWarp, n_last) : 0;
  int p0, p1;
  row_coords<D>(tl, warp, &p0, &p1);
  const int d0 = D == 3 ? nwarps / E1 : nwarps, d1 = D == 3 ? nwarps - d0 * E1 : 0;
#pragma unroll 4
  for (int row = warp; row < rows; row += nwarps) {
    const C* src = gi + row_gbase<D>(geo, o, p0 + p_lo, p1);
    C* dst = tile + (D == 3 ? p0 * PS + p1 * S : p0 * S) + lane;
#pragma unroll
    for (int c = 0; c < NC; ++c)
      if (lane + c * kWarp < E_last) cp_async_elem(dst + c * kWarp, src + col[c]);
    p0 += d0;
    p1 += d1;
    if (D == 3 && p1 >= E1) {
      p1 -= E1;
      ++p0;
    }
  }
  cp_async_wait_all();  // this thread's copies landed; the caller's barrier publishes them
}

// Add the tile into the global grid.  FP32 pairs (even offset on a 16-byte aligned grid
// whose last size is even, so 16-byte aligned and never split by the wrap) go as one
// float4 atomic.  Of `parts` > 1 parts (d <= 2), this call adds part `part`: rows part,
// part + parts, ... (d = 1: pairs of cells).
template <int D, int W, typename C>
__device__ __forceinline__ void flush_tile(const C* tile, C* __restrict__ gi, const Geom& geo, const Tiling& tl,
                                           const TileOrigin& o, int p_lo, int p_n, int part = 0, int parts = 1) {
  constexpr int S = TileShape<D, W, C>::S, PS = TileShape<D, W, C>::PS;
  const int E_last = tl.E[D - 1];
  const int64_t n_last = geo.n[D - 1], a_last = o.a[D - 1];
  const int rows = D == 3 ? p_n * tl.E[1] : (D == 2 ? (tl.E[0] - part + parts - 1) / parts : 1);
  constexpr bool kF32 = sizeof(C) == 8;
  const int tid = threadIdx.x, nt = blockDim.x;
  const bool pairs_ok = kF32 && (n_last & 1) == 0 && (tl.T[D - 1] & 1) == 0 &&  // even tile origin and row length
                       (reinterpret_cast<uintptr_t>(gi) & 15u) == 0;
  const int per_row = pairs_ok ? (E_last + 1) >> 1 : E_last;
  const int total = rows * per_row;
  for (int e = tid; e < total; e += nt) {
    const int row = e / per_row, k = e - row * per_row;
    if (D == 1 && parts > 1 && (pairs_ok ? k : k >> 1) % parts != part) continue;
    int p0, p1;
    row_coords<D>(tl, D == 2 ? part + row * parts : row, &p0, &p1);
    const C* src = tile + (D == 3 ? p0 * PS + p1 * S : (D == 2 ? p0 * S : 0));
    const int64_t gb = row_gbase<D>(geo, o, p0 + p_lo, p1);
    if (pairs_ok) {
      const int p = 2 * k;
      const C v0 = src[p];
      const int64_t gidx = gb + wrap_up(a_last + p, n_last);
      if (p + 1 < E_last) {
        const C v1 = src[p + 1];
        if (v0.x != 0 || v0.y != 0 || v1.x != 0 || v1.y != 0)
          atomicAdd(reinterpret_cast<float4*>(gi + gidx), make_float4(v0.x, v0.y, v1.x, v1.y));
      } else if (v0.x != 0 || v0.y != 0) {
        global_add(gi + gidx, v0);
      }
    } else {
      const C v = src[k];
      if (v.x != 0 || v.y != 0) global_add(gi + gb + wrap_up(a_last + k, n_last), v);
    }
  }
}

// Grab the next work item; returns false when the queue is drained.
__device__ __forceinline__ bool next_item(const Bins& bins, int slot, int4* cur) {
  if (threadIdx.x == 0) {
    const int it = atomicAdd(&bins.work[slot], 1);
    *cur = it < *bins.num_items ? bins.items[it] : make_int4(-1, 0, 0, 0);
  }
  __syncthreads();
  return cur->x >= 0;
}

// CTAs per cluster of the FP32 spreading in 1D and 2D: they take neighbouring items, and add the
// tiles of one grid tile before they go to the grid.
template <int D, typename T>
__host__ __device__ constexpr int spread_cluster() {
  return D < 3 && sizeof(T) == 4 ? 8 : 1;
}
__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive;\n\tbarrier.cluster.wait;" ::: "memory");
}
// what CTA `rank` of the cluster has at this CTA's address p
__device__ __forceinline__ uint32_t cluster_addr(const void* p, int rank) {
  uint32_t a;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"((uint32_t)__cvta_generic_to_shared(p)), "r"(rank));
  return a;
}
__device__ __forceinline__ float2 cluster_load(const float2* p, int rank) {
  float2 v;
  asm volatile("ld.shared::cluster.v2.f32 {%0, %1}, [%2];" : "=f"(v.x), "=f"(v.y) : "r"(cluster_addr(p, rank)) : "memory");
  return v;
}
__device__ __forceinline__ int cluster_load(const int* p, int rank) {
  int v;
  asm volatile("ld.shared::cluster.s32 %0, [%1];" : "=r"(v) : "r"(cluster_addr(p, rank)) : "memory");
  return v;
}

// Shared-memory bytes beyond the tile, per kernel kind (the host sizes launches with it).
__host__ __device__ constexpr int nodes_per_warp_batch(int d) { return d == 1 ? 32 : (d == 2 ? 8 : 4); }
constexpr int kNodesPerCtaBatch = 16;

__host__ __device__ inline size_t grid_extra_smem(int d, int W, size_t real, int nwarps, size_t tile_bytes,
                                                  bool spread) {
  if (!spread) {
    const int nb = nodes_per_warp_batch(d);
    return (size_t)nwarps * ((size_t)nb * d * W * real + (size_t)nb * 2 * sizeof(int));
  }
  // two batch buffers: weights, values, offsets
  const size_t batch = (size_t)kNodesPerCtaBatch * d * W * real + (size_t)kNodesPerCtaBatch * (sizeof(int) + 2 * real);
  return (d == 1 ? (size_t)(nwarps - 1) * tile_bytes : 0) + 2 * batch;
}

// ---------------------------------------------------------------------------
// Interpolation, d = 1..3
// ---------------------------------------------------------------------------
template <int D, int W, typename T>
__global__ void __launch_bounds__(sizeof(T) == 8 || (D == 3 && W > 16) ? 256 : 512) k_interp(const typename Cx<T>::t* __restrict__ g,
                                                typename Cx<T>::t* __restrict__ f, Geom geo, Tiling tl, Bins bins) {
  using C = typename Cx<T>::t;
  constexpr int R = kWarp / W;           // rows (d >= 2) or nodes (d = 1) per warp pass
  constexpr int NIT = (W + R - 1) / R;   // passes over the W rows of a plane
  constexpr bool FULL = R * NIT == W;    // every lane's every pass is a real row
  constexpr int NB = nodes_per_warp_batch(D);
  constexpr int SH = off_bits(D);
  constexpr uint32_t MASK = (1u << SH) - 1u;
  constexpr int S = TileShape<D, W, C>::S, PS = TileShape<D, W, C>::PS;
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ int4 cur;
  C* tile = reinterpret_cast<C*>(smem);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
  T* wb = reinterpret_cast<T*>(smem + tl.smem_tile) + warp * (NB * D * W);
  int* nrec = reinterpret_cast<int*>(reinterpret_cast<T*>(smem + tl.smem_tile) + nwarps * (NB * D * W)) + warp * 2 * NB;
  const int r = lane / W, l_last = lane - r * W;
  const bool lane_on = r < R;
  const T* sfrac = reinterpret_cast<const T*>(bins.sfrac);
  const T norm = (T)geo.norm;
  const int qd = lane / D, td = lane - qd * D;  // (node, dim) of this lane in the weight pass
  // d = 3, W > 16 (and slabs): lane i takes cells i, i + 32, ... of a plane's W x W window, so that
  // no lane idles where W does not divide 32 (bank i mod 16, as S == W mod 16)
  constexpr bool SLAB = TileShape<D, W, C>::SLAB;
  constexpr bool FLAT = D == 3 && (R == 1 || SLAB);
  constexpr int NF = FLAT ? (W * W + kWarp - 1) / kWarp : 1;
  int fcell[NF];
#pragma unroll
  for (int i = 0; i < NF; ++i) {
    const int c = min(lane + i * kWarp, W * W - 1);
    fcell[i] = (c / W) * S + c % W;
  }

  while (next_item(bins, 0, &cur)) {
    const int4 item = cur;
    const TileOrigin o = decode_tile<D>(geo, tl, item.x);
    // nodes per warp and batch: every warp has as many batches, as full as the next one's
    const int per = (item.z - item.y + nwarps - 1) / nwarps, nbat = (per + NB - 1) / NB;
    const int nbw = (per + nbat - 1) / nbat;
    for (int p_lo = 0; p_lo < (SLAB ? tl.E[0] : 1); p_lo += SLAB ? tl.slab : 1) {
      const int p_n = SLAB ? min(tl.slab, tl.E[0] - p_lo) : tl.E[0];
      load_tile<D, W, C>(tile, g + o.inst * geo.ntot, geo, tl, o, p_lo, p_n);
      // records of this warp's first batch
      int bs = item.y + warp * nbw;
      int pf_idx = 0, pf_off = 0;
      T pf_fr = 0;
      if (bs < item.z) {
        const int nb0 = min(nbw, item.z - bs);
        if (lane < nb0) {
          pf_idx = bins.sidx[bs + lane];
          pf_off = bins.soff[bs + lane];
        }
        if (qd < nb0) pf_fr = sfrac[(int64_t)(bs + qd) * D + td];
      }
      __syncthreads();
      for (; bs < item.z; bs += nwarps * nbw) {
        const int nb = min(nbw, item.z - bs);
        if (lane < nb) {
          nrec[lane] = pf_idx;
          nrec[NB + lane] = pf_off;
        }
        if constexpr (sizeof(T) == 8) {
          if (qd < nb) WeightMath<T>::taps(pf_fr, geo.m, geo, td, W, wb + (qd * D + td) * W);
        } else {
          for (int qt0 = 0; qt0 < nb * D; qt0 += R) {
            const int qt = qt0 + r;
            const float fr = __shfl_sync(0xffffffffu, pf_fr, min(qt, 31));
            if (lane_on && qt < nb * D) wb[qt * W + l_last] = WeightMath<T>::tap(fr + (float)(geo.m - l_last), geo, qt % D);
          }
        }
        // fetch the next batch's records while this batch runs
        const int bn = bs + nwarps * nbw;
        if (bn < item.z) {
          const int nbn = min(nbw, item.z - bn);
          if (lane < nbn) {
            pf_idx = bins.sidx[bn + lane];
            pf_off = bins.soff[bn + lane];
          }
          if (qd < nbn) pf_fr = sfrac[(int64_t)(bn + qd) * D + td];
        }
        __syncwarp();
        if (D == 1) {
          for (int q0 = 0; q0 < nb; q0 += R) {
            const int q = q0 + r;
            const bool on = lane_on && q < nb;
            const int qq = on ? q : q0;
            const int o0 = nrec[NB + qq] & MASK;
            C acc = on ? cscale(tile[o0 + l_last], wb[qq * W + l_last]) : czero<C>();
#pragma unroll
            for (int s = 1; s < W; s <<= 1) {
              C o2;
              o2.x = __shfl_down_sync(0xffffffffu, acc.x, s);
              o2.y = __shfl_down_sync(0xffffffffu, acc.y, s);
              if (l_last + s < W) {
                acc.x += o2.x;
                acc.y += o2.y;
              }
            }
            if (on && l_last == 0) f[nrec[qq]] = cscale(acc, norm);
          }
        } else {
          // four nodes at a time: their lane sums are reduced together, each exchange halving
          // what a lane holds (nodes, then components)
          for (int q0 = 0; q0 < nb; q0 += 4) {
            C accs[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) {
              const int q = q0 + u;
              C acc = czero<C>();
              if (FLAT && q < nb) {
                const uint32_t off = (uint32_t)nrec[NB + q];
                const T* wq = wb + q * D * W;
                const int o0 = off & MASK, o1 = (off >> SH) & MASK, o2 = off >> (D == 3 ? 2 * SH : 0);
                const C* tb = tile + (o0 - p_lo) * PS + o1 * S + o2;
                const int lo = SLAB ? max(0, p_lo - o0) : 0, hi = SLAB ? min(W, p_lo + p_n - o0) : W;  // planes of the slab
                C ra[NF];
#pragma unroll
                for (int i = 0; i < NF; ++i) ra[i] = czero<C>();
#pragma unroll 2
                for (int l0 = lo; l0 < hi; ++l0) {
                  const typename WPair<T>::t w0 = WPair<T>::make(wq[l0]);
#pragma unroll
                  for (int i = 0; i < NF; ++i) ra[i] = cmul_addp(ra[i], w0, tb[l0 * PS + fcell[i]]);
                }
#pragma unroll
                for (int i = 0; i < NF; ++i) {
                  const int c = min(lane + i * kWarp, W * W - 1);
                  const T w12 = wq[(D - 2) * W + c / W] * wq[(D - 1) * W + c % W];
                  if (i * kWarp + kWarp <= W * W || lane + i * kWarp < W * W) acc = cmul_add(acc, w12, ra[i]);
                }
              } else if (q < nb && lane_on) {
                const uint32_t off = (uint32_t)nrec[NB + q];
                const T* wq = wb + q * D * W;
                T wrow[NIT];
#pragma unroll
                for (int it = 0; it < NIT; ++it) {
                  const int lr = r + it * R;
                  wrow[it] = (FULL || lr < W) ? wq[(D - 2) * W + (FULL ? lr : min(lr, W - 1))] : (T)0;
                }
                typename WPair<T>::t wpl[D == 3 ? W : 1];
                if (D == 3) {
#pragma unroll
                  for (int l0 = 0; l0 < W; ++l0) wpl[l0] = WPair<T>::make(wq[l0]);
                }
                int base;
                if (D == 3) {
                  const int o0 = off & MASK, o1 = (off >> SH) & MASK, o2 = off >> (D == 3 ? 2 * SH : 0);
                  base = o0 * PS + (o1 + r) * S + o2 + l_last;
                } else {
                  const int o0 = off & MASK, o1 = (off >> SH) & MASK;
                  base = (o0 + r) * S + o1 + l_last;
                }
                const C* tb = tile + base;
#pragma unroll
                for (int it = 0; it < NIT; ++it) {
                  if (FULL || r + it * R < W) {
                    C ra;
                    if (D == 3) {
                      ra = czero<C>();
#pragma unroll
                      for (int l0 = 0; l0 < W; ++l0) ra = cmul_addp(ra, wpl[l0], tb[it * R * S + l0 * PS]);
                    } else {
                      ra = tb[it * R * S];
                    }
                    acc = cmul_add(acc, wrow[it], ra);
                  }
                }
                acc = cscale(acc, wq[(D - 1) * W + l_last]);
              }
              accs[u] = acc;
            }
            __syncwarp();
            const bool h16 = lane & 16, h8 = lane & 8, h4 = lane & 4;
#pragma unroll
            for (int u = 0; u < 2; ++u) {
              const C o2 = shfl_xor_c<C>(h16 ? accs[u] : accs[u + 2], 16);
              const C a = h16 ? accs[u + 2] : accs[u];
              accs[u].x = a.x + o2.x;
              accs[u].y = a.y + o2.y;
            }
            const C o2 = shfl_xor_c<C>(h8 ? accs[0] : accs[1], 8), a = h8 ? accs[1] : accs[0];
            const T ax = a.x + o2.x, ay = a.y + o2.y;
            T v = (h4 ? ay : ax) + __shfl_xor_sync(0xffffffffu, h4 ? ax : ay, 4);
            v += __shfl_xor_sync(0xffffffffu, v, 2);
            v += __shfl_xor_sync(0xffffffffu, v, 1);
            const int q = q0 + (h16 ? 2 : 0) + (h8 ? 1 : 0);
            if ((lane & 3) == 0 && q < nb) {
              T* dst = reinterpret_cast<T*>(f + nrec[q]) + (h4 ? 1 : 0);
              *dst = SLAB && p_lo > 0 ? *dst + v * norm : v * norm;
            }
          }
        }
        __syncwarp();
      }
      __syncthreads();
    }
  }
}

// ---------------------------------------------------------------------------
// Spreading, d = 1..3
// ---------------------------------------------------------------------------
template <int D, int W, typename T>
__global__ void __launch_bounds__(sizeof(T) == 8 ? 256 : 512) k_spread(const typename Cx<T>::t* __restrict__ f,
                                                typename Cx<T>::t* __restrict__ g, Geom geo, Tiling tl, Bins bins) {
  using C = typename Cx<T>::t;
  constexpr int R = kWarp / W;
  constexpr int NIT = (W + R - 1) / R;
  constexpr bool FULL = R * NIT == W;
  constexpr int NBC = kNodesPerCtaBatch;
  constexpr int SH = off_bits(D);
  constexpr uint32_t MASK = (1u << SH) - 1u;
  constexpr int S = TileShape<D, W, C>::S, PS = TileShape<D, W, C>::PS;
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ int4 cur;
  C* tile = reinterpret_cast<C*>(smem);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
  constexpr bool SLAB = TileShape<D, W, C>::SLAB;
  const int tile_elems = D == 1 ? tl.E[0] : (D == 2 ? tl.E[0] * S : tl.slab * PS);
  // d = 1: one private tile copy per warp (copy 0 is `tile`)
  const size_t extra = D == 1 ? (size_t)(nwarps - 1) * tl.smem_tile : 0;
  unsigned char* bptr = smem + tl.smem_tile + extra;
  const size_t batch_bytes = (size_t)NBC * D * W * sizeof(T) + (size_t)NBC * (sizeof(int) + sizeof(C));
  const int r = lane / W, l_last = lane - r * W;
  const bool lane_on = r < R;
  const T* sfrac = reinterpret_cast<const T*>(bins.sfrac);
  const T norm = (T)geo.norm;
  C* mytile = D == 1 ? reinterpret_cast<C*>(smem + (size_t)warp * tl.smem_tile) : tile;
  // this thread's staging role: (node, dim) for weights, node for records
  const int sq = threadIdx.x / D, st = threadIdx.x - sq * D;

  // CL > 1: the cluster's CTAs take CL neighbouring items at a time.  CTA 0 draws the next group
  // while the present one runs; the barriers of a group publish it.
  constexpr int CL = spread_cluster<D, T>();
  const int rank = CL > 1 ? (int)(blockIdx.x % CL) : 0, num = CL > 1 ? *bins.num_items : 0;
  __shared__ int s_next[2];
  auto draw = [&](int slot) {
    if (rank == 0 && threadIdx.x == 0) s_next[slot] = atomicAdd(&bins.work[1], CL);
  };
  if constexpr (CL > 1) {
    draw(0);
    cluster_sync();
  }
  for (int turn = 0;; turn ^= 1) {
    int4 item;
    int valid = 1;      // items of the group
    bool same = false;  // of one tile
    if constexpr (CL > 1) {
      const int base = cluster_load(&s_next[turn], 0);
      if (base >= num) break;
      draw(turn ^ 1);
      valid = min(CL, num - base);
      const int t = bins.items[base + min(lane & (CL - 1), valid - 1)].x, t0 = __shfl_sync(0xffffffffu, t, 0);
      same = valid > 1 && __all_sync(0xffffffffu, t == t0);
      item = rank < valid ? bins.items[base + rank] : make_int4(t0, 0, 0, 0);
    } else {
      if (!next_item(bins, 1, &cur)) break;
      item = cur;
    }
    const TileOrigin o = decode_tile<D>(geo, tl, item.x);
    for (int p_lo = 0; p_lo < (SLAB ? tl.E[0] : 1); p_lo += SLAB ? tl.slab : 1) {
      const int p_n = SLAB ? min(tl.slab, tl.E[0] - p_lo) : tl.E[0];
      {
        const C z = czero<C>();
        if (D == 1) {
          for (int e = lane; e < tile_elems; e += kWarp) mytile[e] = z;
        } else {
          for (int e = threadIdx.x; e < tile_elems; e += blockDim.x) tile[e] = z;
        }
      }
      // records of the first batch
      T pf_fr = 0;
      int pf_off = 0;
      C pf_val = czero<C>();
      {
        const int nb0 = min(NBC, item.z - item.y);
        if (sq < nb0) pf_fr = sfrac[(int64_t)(item.y + sq) * D + st];
        if ((int)threadIdx.x < nb0) {
          pf_off = bins.soff[item.y + threadIdx.x];
          pf_val = f[bins.sidx[item.y + threadIdx.x]];
        }
      }
      int buf = 0;
      for (int bs = item.y; bs < item.z; bs += NBC, buf ^= 1) {
        const int nb = min(NBC, item.z - bs);
        unsigned char* bb = bptr + buf * batch_bytes;
        T* cw = reinterpret_cast<T*>(bb);                      // [NBC][D][W]
        C* cval = reinterpret_cast<C*>(cw + NBC * D * W);      // [NBC]
        int* coff = reinterpret_cast<int*>(cval + NBC);        // [NBC]
        if (sq < nb) WeightMath<T>::taps(pf_fr, geo.m, geo, st, W, cw + (sq * D + st) * W);
        if ((int)threadIdx.x < nb) {
          coff[threadIdx.x] = pf_off;
          cval[threadIdx.x] = cscale(pf_val, norm);
        }
        // fetch the next batch's records
        const int bn = bs + NBC;
        if (bn < item.z) {
          const int nbn = min(NBC, item.z - bn);
          if (sq < nbn) pf_fr = sfrac[(int64_t)(bn + sq) * D + st];
          if ((int)threadIdx.x < nbn) {
            pf_off = bins.soff[bn + threadIdx.x];
            pf_val = f[bins.sidx[bn + threadIdx.x]];
          }
        }
        __syncthreads();  // batch staged (and, for the first batch, the tile cleared)
        if (D == 1) {
          // warp w takes nodes w, w + nwarps, ...; lanes are the node's taps
          for (int q = warp; q < nb; q += nwarps) {
            const int o0 = coff[q] & MASK;
            if (lane < W) {
              C* p = mytile + o0 + lane;
              *p = cmul_add(*p, cw[q * W + lane], cval[q]);
            }
          }
        } else if (D == 2) {
          // warp w owns the row groups {g : g % nwarps == w}, group g = rows g*R .. g*R+R-1
          for (int q = 0; q < nb; ++q) {
            const uint32_t off = (uint32_t)coff[q];
            const int o0 = off & MASK, o1 = (off >> SH) & MASK;
            const int g_first = o0 / R, g_last = (o0 + W - 1) / R;
            const int g0 = g_first + ((warp - g_first % nwarps) + nwarps) % nwarps;
            if (g0 > g_last || !lane_on) continue;
            const T* wq = cw + q * 2 * W;
            const C v = cscale(cval[q], wq[W + l_last]);
            C* tb = tile + o1 + l_last;
            for (int gg = g0; gg <= g_last; gg += nwarps) {
              const int p0 = gg * R + r;
              if (p0 >= o0 && p0 < o0 + W) {
                C* p = tb + p0 * S;
                *p = cmul_add(*p, wq[p0 - o0], v);
              }
            }
          }
        } else {
          // warp w owns the planes {p : p % nwarps == w}
          for (int q = 0; q < nb; ++q) {
            const uint32_t off = (uint32_t)coff[q];
            const int o0 = off & MASK, o1 = (off >> SH) & MASK, o2 = off >> (D == 3 ? 2 * SH : 0);
            const int p_first = SLAB ? max(o0, p_lo) : o0, p_end = SLAB ? min(o0 + W, p_lo + p_n) : o0 + W;
            int p = p_first + ((warp - p_first % nwarps) + nwarps) % nwarps;
            if (p >= p_end || !lane_on) continue;
            const T* wq = cw + q * 3 * W;
            const C v = cscale(cval[q], wq[2 * W + l_last]);
            C vr[NIT];
#pragma unroll
            for (int it = 0; it < NIT; ++it) {
              const int l1 = r + it * R;
              vr[it] = cscale(v, (FULL || l1 < W) ? wq[W + (FULL ? l1 : min(l1, W - 1))] : (T)0);
            }
            C* tb = tile + (o1 + r) * S + o2 + l_last;
            for (; p < p_end; p += nwarps) {
              const typename WPair<T>::t w0 = WPair<T>::make(wq[p - o0]);
              C* tp = tb + (p - p_lo) * PS;
#pragma unroll
              for (int it = 0; it < NIT; ++it) {
                if (FULL || r + it * R < W) {
                  C* t = tp + it * R * S;
                  *t = cmul_addp(*t, w0, vr[it]);
                }
              }
            }
          }
        }
      }
      __syncthreads();
      if (D == 1) {
        // fold the private copies into copy 0, then flush
        for (int e = threadIdx.x; e < tile_elems; e += blockDim.x) {
          C s = tile[e];
          for (int w = 1; w < nwarps; ++w) {
            const C v = reinterpret_cast<const C*>(smem + (size_t)w * tl.smem_tile)[e];
            s.x += v.x;
            s.y += v.y;
          }
          tile[e] = s;
        }
        __syncthreads();
      }
      if constexpr (CL > 1) {
        cluster_sync();
        if (same) {  // this CTA's part of the sum over the cluster's tiles, in place
          const int rows = D == 2 ? (tl.E[0] - rank + CL - 1) / CL : 1;
          const int cols = D == 2 ? tl.E[1] : tl.E[0];
          for (int e = threadIdx.x; e < rows * cols; e += blockDim.x) {
            const int row = e / cols, c = e - row * cols;
            if (D == 1 && (c >> 1) % CL != rank) continue;
            C* const p = tile + (D == 2 ? (rank + row * CL) * S : 0) + c;
            C v = cluster_load(p, 0);
            for (int q = 1; q < valid; ++q) {
              const C w = cluster_load(p, q);
              v.x += w.x;
              v.y += w.y;
            }
            *p = v;
          }
          __syncthreads();
        }
        if (same) flush_tile<D, W, C>(tile, g + o.inst * geo.ntot, geo, tl, o, p_lo, p_n, rank, CL);
        else if (rank < valid) flush_tile<D, W, C>(tile, g + o.inst * geo.ntot, geo, tl, o, p_lo, p_n);
        cluster_sync();  // every tile read before it is cleared
      } else {
        flush_tile<D, W, C>(tile, g + o.inst * geo.ntot, geo, tl, o, p_lo, p_n);
        __syncthreads();
      }
    }
  }
  if constexpr (CL > 1) cluster_sync();  // CTA 0's last draw has been read
}

// One node through global memory: interpolation of the grid at the node (out[idx] written)
// or its sample added to the grid with atomics.  off: the packed tile-local window start,
// fr: the node's D fractions.
template <int D, typename T, bool SPREAD>
__device__ __forceinline__ void grid_node_global(const typename Cx<T>::t* __restrict__ in,
                                                 typename Cx<T>::t* __restrict__ out, const Geom& geo,
                                                 const TileOrigin& o, int idx, uint32_t off,
                                                 const T* __restrict__ fr) {
  using C = typename Cx<T>::t;
  const int W = geo.W;
  const T norm = (T)geo.norm;
  int64_t s[kMaxDim];
  T w[kMaxDim][kMaxTaps];
  for (int t = 0; t < D; ++t) {
    s[t] = o.a[t] + ((off >> (off_bits(D) * t)) & ((1u << off_bits(D)) - 1u));
    WeightMath<T>::taps(fr[t], geo.m, geo, t, W, w[t]);
  }
  const int64_t inst_base = o.inst * geo.ntot;
  if (!SPREAD) {
    C acc;
    acc.x = (T)0;
    acc.y = (T)0;
    for (int l0 = 0; l0 < W; ++l0) {
      const int64_t i0 = wrap_up(s[0] + l0, geo.n[0]);
      if (D == 1) {
        acc = cmul_add(acc, w[0][l0], in[inst_base + i0]);
        continue;
      }
      C a1;
      a1.x = (T)0;
      a1.y = (T)0;
      for (int l1 = 0; l1 < W; ++l1) {
        const int64_t i1 = wrap_up(s[1] + l1, geo.n[1]);
        if (D == 2) {
          a1 = cmul_add(a1, w[1][l1], in[inst_base + i0 * geo.n[1] + i1]);
          continue;
        }
        C a2;
        a2.x = (T)0;
        a2.y = (T)0;
        const int64_t rowb = inst_base + (i0 * geo.n[1] + i1) * geo.n[D - 1];
        for (int l2 = 0; l2 < W; ++l2)
          a2 = cmul_add(a2, w[D - 1][l2], in[rowb + wrap_up(s[D - 1] + l2, geo.n[D - 1])]);
        a1 = cmul_add(a1, w[1][l1], a2);
      }
      acc = cmul_add(acc, w[0][l0], a1);
    }
    out[idx] = cscale(acc, norm);
  } else {
    const C v = cscale(in[idx], norm);
    for (int l0 = 0; l0 < W; ++l0) {
      const int64_t i0 = wrap_up(s[0] + l0, geo.n[0]);
      const C v0 = cscale(v, w[0][l0]);
      if (D == 1) {
        global_add(&out[inst_base + i0], v0);
        continue;
      }
      for (int l1 = 0; l1 < W; ++l1) {
        const int64_t i1 = wrap_up(s[1] + l1, geo.n[1]);
        const C v1 = cscale(v0, w[1][l1]);
        if (D == 2) {
          global_add(&out[inst_base + i0 * geo.n[1] + i1], v1);
          continue;
        }
        const int64_t rowb = inst_base + (i0 * geo.n[1] + i1) * geo.n[D - 1];
        for (int l2 = 0; l2 < W; ++l2)
          global_add(&out[rowb + wrap_up(s[D - 1] + l2, geo.n[D - 1])], cscale(v1, w[D - 1][l2]));
      }
    }
  }
}

}  // namespace cg
