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
// Measured at N = 64^2, M = 4096: forward 98 us (one rotation and one product per term, on
// 16 CTAs, before: 2.28 ms), adjoint 90 us (one sincospi per term before: 9.70 ms); two
// operations per term alone take 56 us at the measured rate.
#include "runtime.h"

namespace cg {

constexpr int kNdftChunk = 256;
constexpr int kNdftPairs = 32;   // pairs per block of the last dimension, at most
constexpr int kNdftRowsF = 8;    // forward: rows per thread
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

template <int D>
__global__ void __launch_bounds__(128) k_ndft_forward(const double* __restrict__ x, const double2* __restrict__ fhat,
                                                      double2* __restrict__ f, Geom geo,
                                                      const int32_t* __restrict__ inst_off, NdftRows nr) {
  constexpr int R = kNdftRowsF;
  __shared__ double2 sd[kNdftPairs][R][2];  // a+ + a-, -i (a+ - a-)
  const int inst = blockIdx.y;
  const int64_t j0 = inst_off[inst], j1 = inst_off[inst + 1];
  const double2* fh = fhat + (int64_t)inst * geo.Ntot;
  const int64_t NL = geo.N[D - 1];
  const int half = (int)(nr.B / 2);
  // row groups g0 .. g1 - 1 of this split (partial sums added atomically)
  const int64_t ng = nr.slow * nr.groups, span = (ng + gridDim.z - 1) / gridDim.z;
  const int64_t g0 = (int64_t)blockIdx.z * span, g1 = min(ng, g0 + span);
  for (int64_t jb = j0 + (int64_t)blockIdx.x * blockDim.x; jb < j1; jb += (int64_t)gridDim.x * blockDim.x) {
    const int64_t j = jb + threadIdx.x;
    const bool on = j < j1;
    double xj[D];
#pragma unroll
    for (int t = 0; t < D; ++t) xj[t] = on ? x[j * D + t] : 0.0;
    const double xl = xj[D - 1];
    const double2 first = cis2pi(0.5 * xl), step = cis2pi(xl - rint(xl));
    const double2 rstep = cis2pi(-(D == 1 ? turn((double)nr.B, xl) : xj[D > 1 ? D - 2 : 0]));
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
        rp = cmul(rp, rstep);
      }
    }
    if (on) {
      if (gridDim.z == 1) {
        f[j] = acc;
      } else {
        atomicAdd(&f[j].x, acc.x);
        atomicAdd(&f[j].y, acc.y);
      }
    }
  }
}

template <int D>
__global__ void __launch_bounds__(256) k_ndft_adjoint(const double* __restrict__ x, const double2* __restrict__ f,
                                                      double2* __restrict__ fhat, Geom geo,
                                                      const int32_t* __restrict__ inst_off, NdftRows nr) {
  constexpr int NJ = kNdftNodesA, RB = kNdftRowsA, SEG = 16;
  __shared__ double2 scs[NJ][kNdftPairs];  // cos, sin of a node's pairs
  __shared__ double2 sc[NJ][RB];           // f_j times the row's phase
  const int inst = blockIdx.y, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int64_t j0 = inst_off[inst], j1 = inst_off[inst + 1];
  const int64_t NL = geo.N[D - 1];
  const int half = (int)(nr.B / 2);
  const NdftGroup<D> q = ndft_group<D>(geo, nr, blockIdx.x);
  // nodes of this split (partial sums added atomically)
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
      for (int t = 0; t < D; ++t) xj[t] = x[(c0 + lane) * D + t];
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
  double2* out = fhat + (int64_t)inst * geo.Ntot;
  for (int r = 0; r < 4; ++r) {
    const int rr = warp * 4 + r;
    if (rr >= q.n || lane >= half) continue;
    const int64_t blk = D == 1 ? q.blk + rr : q.blk, row = (q.lead + rr) * (D == 1 ? 0 : NL);
    const int64_t cp = blk * nr.B + half + lane, cm = blk * nr.B + half - 1 - lane;
    const double2 vp = make_double2(A[r].x - Bv[r].y, A[r].y + Bv[r].x), vm = make_double2(A[r].x + Bv[r].y, A[r].y - Bv[r].x);
    auto put = [&](int64_t c, double2 v) {
      if (c >= NL) return;
      if (gridDim.z == 1) {
        out[row + c] = v;
      } else {
        atomicAdd(&out[row + c].x, v.x);
        atomicAdd(&out[row + c].y, v.y);
      }
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
static int ndft_splits(const Plan& p, int64_t blocks, int64_t inner) {
  const int64_t want = (int64_t)p.num_sms * 4;
  if (blocks >= want) return 1;
  int64_t s = (want + blocks - 1) / blocks;
  const int64_t cap = (inner + 4095) / 4096;
  if (s > cap) s = cap;
  if (s > 65535) s = 65535;
  return (int)(s < 1 ? 1 : s);
}

// Blocks of the last dimension as equal as they come, of at most 2 kNdftPairs coefficients.
static NdftRows ndft_rows(const Geom& geo, int per) {
  NdftRows nr;
  const int64_t NL = geo.N[geo.d - 1];
  nr.nblk = (NL + 2 * kNdftPairs - 1) / (2 * kNdftPairs);
  nr.B = (NL + nr.nblk - 1) / nr.nblk;
  nr.B += nr.B & 1;
  nr.nblk = (NL + nr.B - 1) / nr.B;
  nr.fast = geo.d == 1 ? nr.nblk : geo.N[geo.d - 2];
  nr.slow = geo.d == 1 ? 1 : nr.nblk * (geo.d == 3 ? geo.N[0] : 1);
  nr.per = per;
  nr.groups = (nr.fast + per - 1) / per;
  return nr;
}

static int64_t max_nodes(const Plan& p) {
  int64_t m = 0;
  for (int i = 0; i < p.geo.batch; ++i) m = p.M_inst[i] > m ? p.M_inst[i] : m;
  return m;
}

cudaError_t launch_ndft_forward(const Plan& p, const double* x, const void* fhat, void* f, cudaStream_t st) {
  const int64_t maxM = max_nodes(p);
  if (maxM == 0) return cudaSuccess;
  const NdftRows nr = ndft_rows(p.geo, kNdftRowsF);
  const int64_t ng = nr.slow * nr.groups, want = (int64_t)p.num_sms * 6;
  // one warp per CTA until there are enough CTAs to spread evenly over the SMs
  const int threads = (maxM + 127) / 128 * p.geo.batch * ng >= want ? 128 : 32;
  int64_t bx = (maxM + threads - 1) / threads;
  if (bx > (int64_t)p.num_sms * 16) bx = (int64_t)p.num_sms * 16;
  int64_t splits = (want + bx * p.geo.batch - 1) / (bx * p.geo.batch);
  if (splits > ng) splits = ng;
  if (splits > 65535) splits = 65535;
  if (splits > 1) {
    const cudaError_t e = cudaMemsetAsync(f, 0, sizeof(double2) * p.M, st);
    if (e != cudaSuccess) return e;
  }
  const dim3 grid((unsigned)bx, (unsigned)p.geo.batch, (unsigned)splits);
  auto kern = p.geo.d == 1 ? k_ndft_forward<1> : (p.geo.d == 2 ? k_ndft_forward<2> : k_ndft_forward<3>);
  kern<<<grid, threads, 0, st>>>(x, (const double2*)fhat, (double2*)f, p.geo, p.bins.inst_off, nr);
  return cudaGetLastError();
}

cudaError_t launch_ndft_adjoint(const Plan& p, const double* x, const void* f, void* fhat, cudaStream_t st,
                                const int64_t* kidx, int64_t nsel) {
  const int64_t maxM = max_nodes(p);
  if (kidx) {
    if (nsel == 0) return cudaSuccess;
    int64_t bx = (nsel + 255) / 256;
    if (bx > (int64_t)p.num_sms * 8) bx = (int64_t)p.num_sms * 8;
    const int splits = ndft_splits(p, bx * p.geo.batch, maxM);
    if (splits > 1) {
      const cudaError_t e = cudaMemsetAsync(fhat, 0, sizeof(double2) * nsel * p.geo.batch, st);
      if (e != cudaSuccess) return e;
    }
    const dim3 grid((unsigned)bx, (unsigned)p.geo.batch, (unsigned)splits);
    k_ndft_adjoint_at<<<grid, 256, 0, st>>>(x, (const double2*)f, (double2*)fhat, p.geo, p.bins.inst_off, kidx, nsel);
    return cudaGetLastError();
  }
  const NdftRows nr = ndft_rows(p.geo, kNdftRowsA);
  const int64_t ng = nr.slow * nr.groups;
  // nodes split so that two CTAs run per SM, at least four nodes each
  int64_t splits = (int64_t)p.num_sms * 2 / (ng * p.geo.batch);
  if (splits > (maxM + 3) / 4) splits = (maxM + 3) / 4;
  if (splits < 1) splits = 1;
  if (splits > 1) {
    const cudaError_t e = cudaMemsetAsync(fhat, 0, sizeof(double2) * p.geo.Ntot * p.geo.batch, st);
    if (e != cudaSuccess) return e;
  }
  const dim3 grid((unsigned)ng, (unsigned)p.geo.batch, (unsigned)splits);
  auto kern = p.geo.d == 1 ? k_ndft_adjoint<1> : (p.geo.d == 2 ? k_ndft_adjoint<2> : k_ndft_adjoint<3>);
  kern<<<grid, 256, 0, st>>>(x, (const double2*)f, (double2*)fhat, p.geo, p.bins.inst_off, nr);
  return cudaGetLastError();
}

}  // namespace cg
