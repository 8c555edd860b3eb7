// kernels_ndft.cu -- direct NDFT and adjoint NDFT (FP64), shared-memory staged.
//
// Reference: src/cunfft_kernel.cu:1207-1345 (one thread per output, coefficients
// or nodes read from global memory, cos/sin per term).
//   forward  f_j   = sum_k f_hat_k e^{-2 pi i k.x_j}
//   adjoint  f_hat_k = sum_j f_j   e^{+2 pi i k.x_j}
// with k_t in [-N_t/2, N_t - N_t/2), lexicographic k (last dimension fastest).
//
// GB300 form.  Everything is FP64-pipe work (about 2 multiply-adds per clock and SM), so the
// kernels spend as few operations per (node, coefficient) term as they can.  The last
// dimension is cut into blocks of B <= 64 coefficients around a half-integer centre kc, whose
// coefficients pair up as kc +- (p + 1/2); with phi = 2 pi (p + 1/2) x and the row's phase
// rho (centre and leading dimensions) left to the end,
//   forward   a+ e^{-i phi} + a- e^{i phi} = (a+ + a-) cos phi + (-i)(a+ - a-) sin phi,
//   adjoint   out(+-) = sum_j C cos phi +- i sum_j C sin phi,  C = f_j e^{i rho},
// four real multiply-adds for two complex terms.  The phases of a node are shared by the
// rows (forward: 8 rows of a thread) or computed once per CTA (adjoint: a product over the
// nodes of 32 rows by 32 pairs, 4 rows by 1 pair per thread); they come from sincospi of the
// exactly reduced argument, followed by at most 31 (forward) or 15 (adjoint) rotations.
// Measured at N = 64^2, M = 4096: forward 82 us (one rotation and one product per term, on
// 16 CTAs, before: 2.28 ms), adjoint 69 us (one sincospi per term before: 9.70 ms); two
// operations per term alone take 56 us at the measured rate.
//
// Sums that are split over CTAs go through a buffer of partial sums (at most some 10 MB, kept
// by the plan) and are added in a fixed order, so that results repeat bit by bit: 153 us for
// both directions at N = 64^2, M = 4096, 140 with atomic additions.  A result that is not finite
// is summed again term by term: the sums and differences of pairs turn infinities into NaN, and
// overflow before the terms do.
#include <algorithm>

#include "runtime.h"

namespace cg {

constexpr int kNdftChunk = 256;
constexpr int kNdftPairs = 32;   // pairs per block of the last dimension, at most
constexpr int kNdftRowsF = 8;    // forward: rows per thread, where there are more than two
constexpr int kNdftRowsA = 32;   // adjoint: rows per CTA (4 per warp)
constexpr int kNdftNodesA = 32;  // adjoint: nodes per stage

// Rows of the coefficient array: (block of the last dimension, leading indices), the last
// leading index running fastest (d = 1: the block).
struct NdftRows {
  int64_t B;       // coefficients per block (even)
  int64_t nblk;    // blocks of the last dimension
  int64_t fast;    // rows along the fastest index
  int64_t slow;    // combinations of the others
  int64_t groups;  // groups of consecutive rows along the fastest index
  int64_t per;     // rows per group
  int xs;          // doubles from a node's coordinates to the next one's
};

__device__ __forceinline__ double2 cfma(double2 a, double2 b, double2 acc) {
  acc.x = fma(a.x, b.x, fma(-a.y, b.y, acc.x));
  acc.y = fma(a.x, b.y, fma(a.y, b.x, acc.y));
  return acc;
}

__device__ __forceinline__ double2 cmul(double2 a, double2 b) {
  return make_double2(fma(a.x, b.x, -a.y * b.y), fma(a.x, b.y, a.y * b.x));
}

// k x minus its nearest integer, for k exact in FP64: the product's rounding error is kept
__device__ __forceinline__ double turn(double k, double x) {
  const double p = k * x;
  return (p - rint(p)) + fma(k, x, -p);
}

__device__ __forceinline__ double2 cis2pi(double t) {  // e^{2 pi i t}
  double s, c;
  sincospi(2.0 * t, &s, &c);
  return make_double2(c, s);
}

// First row of a group: its place among the rows, its centre and leading frequencies.
template <int D>
struct NdftGroup {
  int64_t f0;       // first index along the fastest dimension
  int n;            // rows of the group
  int64_t lead;     // index of the first row among the leading dimensions (d > 1)
  int64_t blk;      // its block
  double k[3];      // frequencies of its phase: leading dimensions, then the block's centre
};

template <int D>
__device__ __forceinline__ NdftGroup<D> ndft_group(const Geom& geo, const NdftRows& nr, int64_t g) {
  NdftGroup<D> q;
  const int64_t s = g / nr.groups;
  q.f0 = (g - s * nr.groups) * nr.per;
  q.n = (int)min(nr.per, nr.fast - q.f0);
  q.lead = 0;
  if (D == 1) {
    q.blk = q.f0;
  } else {
    const int64_t outer = D == 3 ? geo.N[0] : 1;  // s = blk * outer + k0 (d = 3), blk (d = 2)
    q.blk = s / outer;
    const int64_t i0 = s - q.blk * outer;
    q.lead = i0 * nr.fast + q.f0;
    if (D == 3) q.k[0] = (double)(i0 - geo.N[0] / 2);
    q.k[D - 2] = (double)(q.f0 - geo.N[D - 2] / 2);
  }
  q.k[D - 1] = (double)(q.blk * nr.B - geo.N[D - 1] / 2) + 0.5 * (double)(nr.B - 1);
  return q;
}

// Phase (turns) of a group's first row at a node; the next row adds the fast dimension's step
template <int D>
__device__ __forceinline__ double ndft_turn(const NdftGroup<D>& q, const double* x) {
  double t = 0.0;
#pragma unroll
  for (int i = 0; i < D; ++i) t += turn(q.k[i], x[i]);
  return t;
}

__device__ __forceinline__ bool finite2(double2 v) { return isfinite(v.x) && isfinite(v.y); }

// f_j term by term
template <int D>
__device__ __noinline__ double2 ndft_node(const Geom& geo, const double2* __restrict__ fh, const double* __restrict__ x) {
  double2 acc = make_double2(0.0, 0.0);
  for (int64_t i = 0; i < geo.Ntot; ++i) {
    double t = 0.0;
    int64_t rem = i;
#pragma unroll
    for (int s = D - 1; s >= 0; --s) {
      t += turn((double)(rem % geo.N[s] - geo.N[s] / 2), x[s]);
      rem /= geo.N[s];
    }
    acc = cfma(fh[i], cis2pi(-t), acc);
  }
  return acc;
}

// coefficient i of an instance term by term
template <int D>
__device__ __noinline__ double2 ndft_coef(const Geom& geo, const double* __restrict__ x, int xs, const double2* __restrict__ f,
                                          int64_t j0, int64_t j1, int64_t i) {
  double k[D];
#pragma unroll
  for (int s = D - 1; s >= 0; --s) {
    k[s] = (double)(i % geo.N[s] - geo.N[s] / 2);
    i /= geo.N[s];
  }
  double2 acc = make_double2(0.0, 0.0);
  for (int64_t j = j0; j < j1; ++j) {
    double t = 0.0;
#pragma unroll
    for (int s = 0; s < D; ++s) t += turn(k[s], x[j * xs + s]);
    acc = cfma(f[j], cis2pi(t), acc);
  }
  return acc;
}

// Partial sums [splits][n] added in a fixed order (warp w of the CTA adds every eighth split of 32
// results, then the warps' sums); what is not finite again term by term.
template <int D, bool ADJ>
__global__ void __launch_bounds__(256) k_ndft_add(const double* __restrict__ x, const double2* __restrict__ in,
                                                  const double2* __restrict__ part, double2* __restrict__ out, Geom geo,
                                                  const int32_t* __restrict__ inst_off, int64_t n, int splits, int xs) {
  __shared__ double2 sum[8][32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (int64_t e0 = blockIdx.x * (int64_t)32; e0 < n; e0 += (int64_t)gridDim.x * 32) {
    const int64_t e = e0 + lane;
    double2 v = make_double2(0.0, 0.0);
    if (e < n) {
#pragma unroll 8
      for (int s = warp; s < splits; s += 8) {
        const double2 p = part[s * n + e];
        v.x += p.x;
        v.y += p.y;
      }
    }
    sum[warp][lane] = v;
    __syncthreads();
    if (warp == 0 && e < n) {
#pragma unroll
      for (int w = 1; w < 8; ++w) {
        v.x += sum[w][lane].x;
        v.y += sum[w][lane].y;
      }
      if (!finite2(v)) {
        if (ADJ) {
          const int64_t inst = e / geo.Ntot;
          v = ndft_coef<D>(geo, x, xs, in, inst_off[inst], inst_off[inst + 1], e - inst * geo.Ntot);
        } else {
          int inst = 0;
          while (inst + 1 < geo.batch && inst_off[inst + 1] <= e) ++inst;
          v = ndft_node<D>(geo, in + inst * geo.Ntot, x + e * xs);
        }
      }
      out[e] = v;
    }
    __syncthreads();
  }
}

// SPLIT: partial sums of split blockIdx.z to part [split][total], total nodes of all instances
template <int D, int R, bool SPLIT>
__global__ void __launch_bounds__(128) k_ndft_forward(const double* __restrict__ x, const double2* __restrict__ fhat,
                                                      double2* __restrict__ f, Geom geo,
                                                      const int32_t* __restrict__ inst_off, NdftRows nr,
                                                      double2* __restrict__ part, int64_t total) {
  __shared__ double2 sd[kNdftPairs][R][2];  // a+ + a-, -i (a+ - a-)
  const int inst = blockIdx.y;
  const int64_t j0 = inst_off[inst], j1 = inst_off[inst + 1];
  const double2* fh = fhat + (int64_t)inst * geo.Ntot;
  const int64_t NL = geo.N[D - 1];
  const int half = (int)(nr.B / 2);
  // row groups g0 .. g1 - 1 of this split
  const int64_t ng = nr.slow * nr.groups, span = (ng + gridDim.z - 1) / gridDim.z;
  const int64_t g0 = (int64_t)blockIdx.z * span, g1 = min(ng, g0 + span);
  for (int64_t jb = j0 + (int64_t)blockIdx.x * blockDim.x; jb < j1; jb += (int64_t)gridDim.x * blockDim.x) {
    const int64_t j = jb + threadIdx.x;
    const bool on = j < j1;
    double xj[D];
#pragma unroll
    for (int t = 0; t < D; ++t) xj[t] = on ? x[j * nr.xs + t] : 0.0;
    const double xl = xj[D - 1];
    const double2 first = cis2pi(0.5 * xl), step = cis2pi(xl - rint(xl));
    const double2 rstep = R > 1 ? cis2pi(-(D == 1 ? turn((double)nr.B, xl) : xj[D > 1 ? D - 2 : 0])) : first;
    double2 acc = make_double2(0.0, 0.0);
    for (int64_t g = g0; g < g1; ++g) {
      const NdftGroup<D> q = ndft_group<D>(geo, nr, g);
      __syncthreads();
      for (int e = threadIdx.x; e < half * R; e += blockDim.x) {
        const int r = e / half, p = e - r * half;  // consecutive threads along the row
        double2 ap = make_double2(0.0, 0.0), am = ap;
        if (r < q.n) {
          const int64_t blk = D == 1 ? q.blk + r : q.blk, row = (q.lead + r) * (D == 1 ? 0 : NL);
          const int64_t cp = blk * nr.B + half + p, cm = blk * nr.B + half - 1 - p;
          if (cp < NL) ap = fh[row + cp];
          if (cm < NL) am = fh[row + cm];
        }
        sd[p][r][0] = make_double2(ap.x + am.x, ap.y + am.y);
        sd[p][r][1] = make_double2(ap.y - am.y, am.x - ap.x);
      }
      __syncthreads();
      double2 s[R];
#pragma unroll
      for (int r = 0; r < R; ++r) s[r] = make_double2(0.0, 0.0);
      double2 ph = first;
      for (int p = 0; p < half; ++p) {
#pragma unroll
        for (int r = 0; r < R; ++r) {
          const double2 a = sd[p][r][0], b = sd[p][r][1];
          s[r].x = fma(b.x, ph.y, fma(a.x, ph.x, s[r].x));
          s[r].y = fma(b.y, ph.y, fma(a.y, ph.x, s[r].y));
        }
        ph = cmul(ph, step);
      }
      double2 rp = cis2pi(-ndft_turn<D>(q, xj));
#pragma unroll
      for (int r = 0; r < R; ++r) {
        acc = cfma(s[r], rp, acc);
        if (R > 1) rp = cmul(rp, rstep);
      }
    }
    if (on) {
      if (SPLIT) part[blockIdx.z * total + j] = acc;
      else f[j] = finite2(acc) ? acc : ndft_node<D>(geo, fh, x + j * nr.xs);
    }
  }
}

template <int D, bool SPLIT>
__global__ void __launch_bounds__(256) k_ndft_adjoint(const double* __restrict__ x, const double2* __restrict__ f,
                                                      double2* __restrict__ fhat, Geom geo,
                                                      const int32_t* __restrict__ inst_off, NdftRows nr,
                                                      double2* __restrict__ part) {
  constexpr int NJ = kNdftNodesA, RB = kNdftRowsA, SEG = 16;
  __shared__ double2 scs[NJ][kNdftPairs];  // cos, sin of a node's pairs
  __shared__ double2 sc[NJ][RB];           // f_j times the row's phase
  const int inst = blockIdx.y, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int64_t j0 = inst_off[inst], j1 = inst_off[inst + 1];
  const int64_t NL = geo.N[D - 1];
  const int half = (int)(nr.B / 2);
  const NdftGroup<D> q = ndft_group<D>(geo, nr, blockIdx.x);
  // nodes of this split
  const int64_t span = (j1 - j0 + gridDim.z - 1) / gridDim.z;
  const int64_t n_lo = j0 + (int64_t)blockIdx.z * span, n_hi = min(j1, n_lo + span);
  double2 A[4], Bv[4];
#pragma unroll
  for (int r = 0; r < 4; ++r) A[r] = Bv[r] = make_double2(0.0, 0.0);
  for (int64_t c0 = n_lo; c0 < n_hi; c0 += NJ) {
    const int cn = (int)min((int64_t)NJ, n_hi - c0);
    __syncthreads();
    // phases, a segment of SEG of one node per thread: warps 0, 1 the pairs, 2, 3 the rows
    if (warp < 4 && lane < cn) {
      const int lo = (warp & 1) * SEG;
      double xj[D];
#pragma unroll
      for (int t = 0; t < D; ++t) xj[t] = x[(c0 + lane) * nr.xs + t];
      const double xl = xj[D - 1];
      if (warp < 2) {
        if (lo < half) {
          double2 ph = cis2pi(turn((double)lo + 0.5, xl));
          const double2 st = cis2pi(xl - rint(xl));
          for (int p = lo; p < min(half, lo + SEG); ++p) {
            scs[lane][p] = ph;
            ph = cmul(ph, st);
          }
        }
      } else if (lo < q.n) {
        const double fs = D == 1 ? (double)nr.B : 1.0, xf = D == 1 ? xl : xj[D > 1 ? D - 2 : 0];
        double2 ph = cis2pi(ndft_turn<D>(q, xj) + turn(fs * lo, xf));
        ph = cmul(ph, f[c0 + lane]);
        const double2 st = cis2pi(turn(fs, xf));
        for (int r = lo; r < lo + SEG; ++r) {
          sc[lane][r] = ph;
          ph = cmul(ph, st);
        }
      }
    }
    __syncthreads();
    if (warp * 4 < q.n) {
      for (int n = 0; n < cn; ++n) {
        const double2 cs = scs[n][min(lane, half - 1)];
#pragma unroll
        for (int r = 0; r < 4; ++r) {
          const double2 c = sc[n][warp * 4 + r];
          A[r].x = fma(c.x, cs.x, A[r].x);
          A[r].y = fma(c.y, cs.x, A[r].y);
          Bv[r].x = fma(c.x, cs.y, Bv[r].x);
          Bv[r].y = fma(c.y, cs.y, Bv[r].y);
        }
      }
    }
  }
  double2* out = (SPLIT ? part + blockIdx.z * (geo.Ntot * geo.batch) : fhat) + (int64_t)inst * geo.Ntot;
  for (int r = 0; r < 4; ++r) {
    const int rr = warp * 4 + r;
    if (rr >= q.n || lane >= half) continue;
    const int64_t blk = D == 1 ? q.blk + rr : q.blk, row = (q.lead + rr) * (D == 1 ? 0 : NL);
    const int64_t cp = blk * nr.B + half + lane, cm = blk * nr.B + half - 1 - lane;
    const double2 vp = make_double2(A[r].x - Bv[r].y, A[r].y + Bv[r].x), vm = make_double2(A[r].x + Bv[r].y, A[r].y - Bv[r].x);
    auto put = [&](int64_t c, double2 v) {
      if (c >= NL) return;
      out[row + c] = SPLIT || finite2(v) ? v : ndft_coef<D>(geo, x, nr.xs, f, j0, j1, row + c);
    };
    put(cp, vp);
    put(cm, vm);
  }
}

// The nsel coefficient indices kidx[] of instance blockIdx.y, written densely; one
// coefficient per thread, sincospi per term.
__global__ void __launch_bounds__(256) k_ndft_adjoint_at(const double* __restrict__ x, const double2* __restrict__ f,
                                                      double2* __restrict__ fhat, Geom geo,
                                                      const int32_t* __restrict__ inst_off,
                                                      const int64_t* __restrict__ kidx, int64_t nsel) {
  __shared__ double sx[kNdftChunk * kMaxDim];
  __shared__ double2 sf[kNdftChunk];
  const int d = geo.d;
  const int inst = blockIdx.y;
  const int64_t j0 = inst_off[inst], j1 = inst_off[inst + 1];
  const int64_t nout = nsel;
  double2* out = fhat + (int64_t)inst * nout;
  for (int64_t kb = (int64_t)blockIdx.x * blockDim.x; kb < nout; kb += (int64_t)gridDim.x * blockDim.x) {
    const int64_t kl = kb + threadIdx.x;
    const bool on = kl < nout;
    double kk[kMaxDim] = {0.0, 0.0, 0.0};
    if (on) {
      int64_t rem = kidx[kl];
      for (int t = d - 1; t >= 0; --t) {
        kk[t] = (double)(rem % geo.N[t] - geo.N[t] / 2);
        rem /= geo.N[t];
      }
    }
    double2 acc = make_double2(0.0, 0.0);
    // split of the node range over blockIdx.z (partial sums added atomically)
    const int64_t span = ((j1 - j0 + gridDim.z - 1) / gridDim.z + kNdftChunk - 1) / kNdftChunk * kNdftChunk;
    const int64_t n_lo = j0 + (int64_t)blockIdx.z * span, n_hi = min(j1, n_lo + span);
    for (int64_t c0 = n_lo; c0 < n_hi; c0 += kNdftChunk) {
      const int cn = (int)min((int64_t)kNdftChunk, n_hi - c0);
      __syncthreads();
      for (int e = threadIdx.x; e < cn * d; e += blockDim.x) sx[e] = x[c0 * d + e];
      if (threadIdx.x < cn) sf[threadIdx.x] = f[c0 + threadIdx.x];
      __syncthreads();
      for (int s = 0; s < cn; ++s) {
        double kx = 0.0;
        for (int t = 0; t < d; ++t) kx = fma(kk[t], sx[s * d + t], kx);
        double sp, cp;
        sincospi(2.0 * kx, &sp, &cp);
        acc = cfma(sf[s], make_double2(cp, sp), acc);
      }
    }
    if (on) {
      if (gridDim.z == 1) {
        out[kl] = acc;
      } else {
        atomicAdd(&out[kl].x, acc.x);
        atomicAdd(&out[kl].y, acc.y);
      }
    }
  }
}

// Few selected coefficients would occupy a few SMs only: split the inner sum over up to 4 CTAs per SM, at least 4096 terms each.
static int ndft_at_splits(const Plan& p, int64_t blocks, int64_t inner) {
  const int64_t want = (int64_t)p.num_sms * 4;
  if (blocks >= want) return 1;
  int64_t s = (want + blocks - 1) / blocks;
  const int64_t cap = (inner + 4095) / 4096;
  if (s > cap) s = cap;
  if (s > 65535) s = 65535;
  return (int)(s < 1 ? 1 : s);
}

// Blocks of the last dimension as equal as they come, of at most 2 kNdftPairs coefficients.
static NdftRows ndft_rows(const Geom& geo, int per, int xs) {
  NdftRows nr;
  const int64_t NL = geo.N[geo.d - 1];
  nr.nblk = (NL + 2 * kNdftPairs - 1) / (2 * kNdftPairs);
  nr.B = (NL + nr.nblk - 1) / nr.nblk;
  nr.B += nr.B & 1;
  nr.nblk = (NL + nr.B - 1) / nr.B;
  nr.fast = geo.d == 1 ? nr.nblk : geo.N[geo.d - 2];
  nr.slow = geo.d == 1 ? 1 : nr.nblk * (geo.d == 3 ? geo.N[0] : 1);
  nr.per = per;
  nr.xs = xs;
  nr.groups = (nr.fast + per - 1) / per;
  return nr;
}

static int64_t max_nodes(const Plan& p) {
  int64_t m = 0;
  for (int i = 0; i < p.geo.batch; ++i) m = p.M_inst[i] > m ? p.M_inst[i] : m;
  return m;
}

// Launch of one direction: CTAs along nodes (forward) or row groups (adjoint), splits, results.
struct NdftLaunch {
  Geom geo;
  NdftRows nr;
  int threads;
  int64_t bx, splits, results;
};

// The geometry without trailing dimensions of one coefficient (frequency zero), which would leave
// a block with one coefficient: N = 20000 x 1, M = 300 adjoint 1.68 ms, 0.06 as 1D.
static Geom ndft_geom(Geom g) {
  while (g.d > 1 && g.N[g.d - 1] == 1) --g.d;
  return g;
}

static NdftLaunch ndft_launch_forward(const Plan& p) {
  NdftLaunch l;
  const int64_t maxM = max_nodes(p), want = (int64_t)p.num_sms * 6;
  l.geo = ndft_geom(p.geo);
  l.nr = ndft_rows(l.geo, kNdftRowsF, p.geo.d);
  if (l.nr.fast <= 2) l.nr = ndft_rows(l.geo, 1, p.geo.d);  // M = 1e5, N = 4: 66 us with 8 rows per thread, 38 with one; N = 64: 259, 83
  const int64_t ng = l.nr.slow * l.nr.groups;
  // one warp per CTA until there are enough CTAs to spread evenly over the SMs
  l.threads = (maxM + 127) / 128 * p.geo.batch * ng >= want ? 128 : 32;
  l.bx = std::max<int64_t>(1, (maxM + l.threads - 1) / l.threads);
  if (l.bx > (int64_t)p.num_sms * 16) l.bx = (int64_t)p.num_sms * 16;
  l.splits = (want + l.bx * p.geo.batch - 1) / (l.bx * p.geo.batch);
  if (l.splits > ng) l.splits = ng;
  if (l.splits > 65535) l.splits = 65535;
  l.results = p.M;
  return l;
}

static NdftLaunch ndft_launch_adjoint(const Plan& p) {
  NdftLaunch l;
  const int64_t maxM = max_nodes(p);
  l.geo = ndft_geom(p.geo);
  l.nr = ndft_rows(l.geo, kNdftRowsA, p.geo.d);
  l.threads = 256;
  l.bx = l.nr.slow * l.nr.groups;
  // nodes split so that two CTAs run per SM, at least four nodes each
  l.splits = (int64_t)p.num_sms * 2 / (l.bx * p.geo.batch);
  if (l.splits > (maxM + 3) / 4) l.splits = (maxM + 3) / 4;
  if (l.splits < 1) l.splits = 1;
  l.results = p.geo.Ntot * p.geo.batch;
  return l;
}

// Splits of a direction's sums: as planned where the plan has room for the partial sums (made for
// both directions at once), 1 where it cannot be had, and while the stream is captured (the graph
// may outlive the room).
static int64_t ndft_splits(Plan& p, const NdftLaunch& l, cudaStream_t st) {
  if (l.splits <= 1) return 1;
  cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
  if (cudaStreamIsCapturing(st, &cs) != cudaSuccess || cs != cudaStreamCaptureStatusNone) {
    cudaGetLastError();
    return 1;
  }
  if (l.splits * l.results <= p.nd_cap) return l.splits;
  const NdftLaunch f = ndft_launch_forward(p), a = ndft_launch_adjoint(p);
  const int64_t need = std::max(f.splits > 1 ? f.splits * f.results : 0, a.splits > 1 ? a.splits * a.results : 0);
  ndft_release(p);
  if (plan_malloc(&p.nd_part, sizeof(double2) * (size_t)need) != cudaSuccess) {
    cudaGetLastError();
    p.nd_part = nullptr;
    return 1;
  }
  p.nd_cap = need;
  return l.splits;
}

void ndft_release(Plan& p) {
  cudaFree(p.nd_part);
  p.nd_part = nullptr;
  p.nd_cap = 0;
}

template <bool ADJ>
static cudaError_t add_partial_sums(const Plan& p, const NdftLaunch& l, const double* x, const void* in, void* out, int splits,
                                    cudaStream_t st) {
  int64_t blocks = (l.results + 31) / 32;
  if (blocks > (int64_t)p.num_sms * 8) blocks = (int64_t)p.num_sms * 8;
  auto kern = l.geo.d == 1 ? k_ndft_add<1, ADJ> : (l.geo.d == 2 ? k_ndft_add<2, ADJ> : k_ndft_add<3, ADJ>);
  kern<<<(unsigned)blocks, 256, 0, st>>>(x, (const double2*)in, (const double2*)p.nd_part, (double2*)out, l.geo, p.bins.inst_off,
                                         l.results, splits, l.nr.xs);
  return cudaGetLastError();
}

template <int R, bool SPLIT>
static auto ndft_forward_kernel(int d) {
  return d == 1 ? k_ndft_forward<1, R, SPLIT> : (d == 2 ? k_ndft_forward<2, R, SPLIT> : k_ndft_forward<3, R, SPLIT>);
}

cudaError_t launch_ndft_forward(Plan& p, const double* x, const void* fhat, void* f, cudaStream_t st) {
  if (max_nodes(p) == 0) return cudaSuccess;
  const NdftLaunch l = ndft_launch_forward(p);
  const int64_t splits = ndft_splits(p, l, st);
  const dim3 grid((unsigned)l.bx, (unsigned)p.geo.batch, (unsigned)splits);
  auto kern = splits > 1 ? (l.nr.per == 1 ? ndft_forward_kernel<1, true>(l.geo.d) : ndft_forward_kernel<kNdftRowsF, true>(l.geo.d))
                         : (l.nr.per == 1 ? ndft_forward_kernel<1, false>(l.geo.d) : ndft_forward_kernel<kNdftRowsF, false>(l.geo.d));
  kern<<<grid, l.threads, 0, st>>>(x, (const double2*)fhat, (double2*)f, l.geo, p.bins.inst_off, l.nr, (double2*)p.nd_part, p.M);
  if (splits > 1) return add_partial_sums<false>(p, l, x, fhat, f, (int)splits, st);
  return cudaGetLastError();
}

cudaError_t launch_ndft_adjoint(Plan& p, const double* x, const void* f, void* fhat, cudaStream_t st,
                                const int64_t* kidx, int64_t nsel) {
  if (kidx) {
    if (nsel == 0) return cudaSuccess;
    int64_t bx = (nsel + 255) / 256;
    if (bx > (int64_t)p.num_sms * 8) bx = (int64_t)p.num_sms * 8;
    const int splits = ndft_at_splits(p, bx * p.geo.batch, max_nodes(p));
    if (splits > 1) {
      const cudaError_t e = cudaMemsetAsync(fhat, 0, sizeof(double2) * nsel * p.geo.batch, st);
      if (e != cudaSuccess) return e;
    }
    const dim3 grid((unsigned)bx, (unsigned)p.geo.batch, (unsigned)splits);
    k_ndft_adjoint_at<<<grid, 256, 0, st>>>(x, (const double2*)f, (double2*)fhat, p.geo, p.bins.inst_off, kidx, nsel);
    return cudaGetLastError();
  }
  const NdftLaunch l = ndft_launch_adjoint(p);
  const int64_t splits = ndft_splits(p, l, st);
  const dim3 grid((unsigned)l.bx, (unsigned)p.geo.batch, (unsigned)splits);
  auto kern = splits > 1 ? (l.geo.d == 1 ? k_ndft_adjoint<1, true> : (l.geo.d == 2 ? k_ndft_adjoint<2, true> : k_ndft_adjoint<3, true>))
                         : (l.geo.d == 1 ? k_ndft_adjoint<1, false> : (l.geo.d == 2 ? k_ndft_adjoint<2, false> : k_ndft_adjoint<3, false>));
  kern<<<grid, l.threads, 0, st>>>(x, (const double2*)f, (double2*)fhat, l.geo, p.bins.inst_off, l.nr, (double2*)p.nd_part);
  if (splits > 1) return add_partial_sums<true>(p, l, x, f, fhat, (int)splits, st);
  return cudaGetLastError();
}

}  // namespace cg
