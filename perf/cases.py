"""Timed cases of the NFFT library: its workloads through the public entry points.

A case is a dict of plain values.  ``kind`` names the way a program uses the library:

  step      bind a new node set, forward and adjoint transform on device tensors
  graph     adjoint and forward replayed as CUDA graphs on a bound node set
  autograd  differentiable transform: loss, gradients of nodes and coefficients
  cg        inverse NFFT: conjugate gradients on the normal equations
  ndft      direct NDFT and adjoint NDFT
  dropin    the reference's C plan API between host buffers, copies included

``N`` and ``n`` are sizes joined by "x" (``n`` empty: the plan's default, 2 next_pow2(N)).
``exact`` evaluates the same windowed sums (the direct sums for ``ndft``) with torch in
64 bits.
"""
import math

import numpy as np
import torch

from cunfft_gb300.abi import ReferencePlan
from cunfft_gb300.autograd import nfft
from cunfft_gb300.nfft import NFFT
from cunfft_gb300.solver import cgne

DEV = "cuda:0"


def listed():
    return [
        # the reference's test driver at its smallest published 2D size: one program run is copies
        # in, transform, copies out, and the same for the adjoint; latency and launches
        dict(name="dropin 2D 64^2", kind="dropin", N="64x64", n="", m=6, prec="f64", window="gaussian", M=4096, nodes="uniform", batch=1),
        # direct NDFT of the same size, the check that the reference's drivers run beside it
        dict(name="ndft 2D 64^2", kind="ndft", N="64x64", n="", m=6, prec="f64", window="gaussian", M=4096, nodes="uniform", batch=1),
        # long 1D signals, FP64
        dict(name="step 1D 2^17 f64", kind="step", N="131072", n="", m=6, prec="f64", window="gaussian", M=131072, nodes="uniform", batch=1),
        # 2D images in the reference's precision (its published 2D size)
        dict(name="step 2D 512^2 f64", kind="step", N="512x512", n="", m=6, prec="f64", window="gaussian", M=262144, nodes="uniform", batch=1),
        # the reference's published 3D size, m = 6 and its high-accuracy setting m = 12
        dict(name="step 3D 64^3 f64", kind="step", N="64x64x64", n="", m=6, prec="f64", window="gaussian", M=262144, nodes="uniform", batch=1),
        dict(name="step 3D 64^3 f64 m12", kind="step", N="64x64x64", n="", m=12, prec="f64", window="gaussian", M=262144, nodes="uniform", batch=1),
        # the headline size in FP32
        dict(name="step 3D 128^3 f32", kind="step", N="128x128x128", n="", m=6, prec="f32", window="gaussian", M=2097152, nodes="uniform", batch=1),
        # odd bandwidths on grid sizes that are not powers of two, ES window, odd node count
        dict(name="step 3D odd f32 es", kind="step", N="51x38x63", n="110x84x126", m=4, prec="f32", window="es", M=100003, nodes="uniform", batch=1),
        # MRI-like trajectories: radial spokes and a dense centre
        dict(name="step 2D clustered f32", kind="step", N="512x512", n="", m=6, prec="f32", window="gaussian", M=786432, nodes="spokes", batch=1),
        # many transforms of uneven node counts (1e3 to 1e6), replayed on bound nodes
        dict(name="graph 2D batch f32", kind="graph", N="256x256", n="", m=5, prec="f32", window="gaussian", M=105773, nodes="uniform", batch=64),
        # learning node positions and coefficients by gradient descent
        dict(name="autograd 2D 256^2 f32", kind="autograd", N="256x256", n="", m=6, prec="f32", window="gaussian", M=262144, nodes="uniform", batch=1),
        # reconstruction of coefficients from samples, ten iterations
        dict(name="cg 2D 192^2 f32", kind="cg", N="192x192", n="", m=6, prec="f32", window="gaussian", M=150001, nodes="uniform", batch=1),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choices(["step", "dropin", "ndft", "graph", "autograd", "cg"], [10, 2, 2, 2, 2, 1])[0]
    c = dict(kind=kind, n="", m=rng.choice([3, 4, 5, 6, 6, 6, 6, 7, 8, 12]), prec=rng.choice(["f32", "f64"]), window="gaussian", nodes="uniform", batch=1)
    if kind == "ndft":
        d = rng.choice([1, 2, 3])
        N = [_log(rng, *{1: (64, 16384), 2: (16, 128), 3: (8, 32)}[d]) for _ in range(d)]
        M = _log(rng, 64, 16384)
        c["prec"], c["m"] = "f64", 6
    elif kind == "dropin":
        d = rng.choice([1, 2, 3])
        N = [_log(rng, *{1: (16, 65536), 2: (16, 256), 3: (8, 40)}[d]) for _ in range(d)]
        M = _log(rng, 16, 65536)
        c["prec"], c["m"] = "f64", 6
    elif kind == "cg":
        d = rng.choice([1, 2])
        N = [_log(rng, *{1: (64, 16384), 2: (24, 256)}[d]) for _ in range(d)]
        M = 4 * math.prod(N) + rng.randint(0, 999)
        c["m"] = rng.choice([5, 6, 7])
    else:
        d = rng.choices([1, 2, 3], [2, 5, 4])[0]
        hi = {1: 1 << 17, 2: 512, 3: 80}[d]
        N = [_log(rng, *{1: (128, hi), 2: (24, hi), 3: (12, hi)}[d]) for _ in range(d)]
        M = _log(rng, 500, 1 << (19 if d < 3 else 18))
        if kind == "graph":
            c["batch"] = rng.randint(2, 24)
            M = max(8, min(M, 50000))
            N = [min(v, 200 if d == 2 else 40) if d > 1 else min(v, 8192) for v in N]
        if kind != "autograd" and rng.random() < 0.25:
            c["window"] = "es"
        if rng.random() < 0.35:
            c["n"] = "x".join(str(2 * v + rng.randint(0, 9)) for v in N)
        if d == 2 and c["batch"] == 1 and rng.random() < 0.3:
            c["nodes"] = "spokes"
    c["N"], c["M"] = "x".join(map(str, N)), M
    return c


def _sizes(case):
    N = [int(v) for v in case["N"].split("x")]
    if case["n"]:
        n = [int(v) for v in case["n"].split("x")]
    else:
        n = [2 << (v - 1).bit_length() for v in N]
    return N, n


def _counts(case):
    """Nodes per instance: batched plans have uneven counts around M, log-uniform over three decades."""
    if case["batch"] == 1:
        return [case["M"]]
    r = np.random.default_rng(404)
    w = 10.0 ** r.uniform(0, 3, case["batch"])
    return [max(1, int(v)) for v in np.round(w / w.mean() * case["M"])]


def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(int(seed) * 2654435761 % (1 << 62) + 17)


def _nodes(case, M, d, g):
    if case["nodes"] == "uniform":
        return torch.rand(M, d, generator=g, device=DEV, dtype=torch.float64) - 0.5
    # two thirds on radial spokes, one third in a Gaussian blob at the origin
    blob = M // 3
    rad = M - blob
    spokes = max(1, int(math.sqrt(rad / 2)))
    k = torch.arange(rad, device=DEV)
    turn = torch.rand((), generator=g, device=DEV, dtype=torch.float64)
    th = math.pi * ((k % spokes).double() + turn) / spokes
    r = torch.div(k, spokes, rounding_mode="floor").double() / -(-rad // spokes) - 0.5
    a = torch.stack([torch.cos(th) * r, torch.sin(th) * r], 1)
    b = torch.randn(blob, 2, generator=g, device=DEV, dtype=torch.float64) * 0.02
    x = torch.cat([a, b])
    return (x + 0.5 - torch.floor(x + 0.5) - 0.5).contiguous()


def _crand(shape, g, dtype):
    v = torch.rand(*shape, 2, generator=g, device=DEV, dtype=torch.float64) * 2 - 1
    return torch.view_as_complex(v).to(dtype)


def _inputs(case, seed):
    N, _ = _sizes(case)
    g = _gen(seed)
    counts = _counts(case)
    M = sum(counts)
    dtype = torch.complex64 if case["prec"] == "f32" else torch.complex128
    x = _nodes(case, M, len(N), g)
    shape = ([case["batch"]] if case["batch"] > 1 else []) + N
    return x, counts, _crand(shape, g, dtype), _crand([M], g, dtype)


def prepare(case, seed):
    N, n = _sizes(case)
    x, counts, fh, f = _inputs(case, seed)
    s = dict(case=case, x=x, counts=counts, fh=fh, f=f)
    if case["kind"] == "dropin":
        p = ReferencePlan(N, case["M"], m=case["m"])
        p.x[:] = x.cpu().numpy()
        s["fh"] = fh.cpu().numpy().reshape(-1)
        s["plan"] = p
        return s
    p = NFFT(N, n=n if case["n"] else None, m=case["m"], precision=case["prec"], batch=case["batch"], device=DEV,
             window=case["window"])
    s["plan"] = p
    if case["kind"] in ("graph", "cg", "ndft"):
        p.set_nodes(x, counts)
    if case["kind"] == "graph":
        s["of"] = torch.empty_like(f)
        s["ofh"] = torch.empty_like(fh)
    if case["kind"] == "autograd":
        s["x"] = x.requires_grad_(True)
        s["fh"] = fh.requires_grad_(True)
    return s


def run(s):
    p, kind = s["plan"], s["case"]["kind"]
    if kind == "step":
        p.set_nodes(s["x"], s["counts"])
        return [p.forward(s["fh"]), p.adjoint(s["f"])]
    if kind == "graph":
        return [p.adjoint_graph(s["f"], s["ofh"]), p.forward_graph(s["fh"], s["of"])]
    if kind == "autograd":
        y = nfft(s["x"], s["fh"], plan=p)
        loss = (y - s["f"]).abs().square().sum()
        gx, gfh = torch.autograd.grad(loss, (s["x"], s["fh"]))
        return [y.detach(), gx, gfh]
    if kind == "cg":
        return cgne(p, s["f"], iters=10)[0]
    if kind == "ndft":
        return [p.ndft_forward(s["fh"]), p.ndft_adjoint(s["f"])]
    p.f_hat[:] = s["fh"]
    p.copyDataToDevice()
    p.cunfft_transform()
    p.copyDataToHost()
    p.copyDataToDeviceAd()
    p.cunfft_adjoint()
    p.copyDataToHostAd()
    p.check()
    return [p.f.copy(), p.f_hat.copy()]  # the views end with the plan


def work(case):
    N, n = _sizes(case)
    d, B, M = len(N), case["batch"], sum(_counts(case))
    c = 8 if case["prec"] == "f32" else 16
    Nt, nt, taps = math.prod(N) * B, math.prod(n) * B, (2 * case["m"] + 2) ** d
    if case["kind"] == "ndft":
        # one complex multiply-add per (node, coefficient) pair and direction
        return dict(bytes=2 * (8 * d * M + 16 * (M + Nt)), flops=2 * 8.0 * M * Nt)
    # per direction: nodes, coefficients and samples once; an FFT, and a complex-by-real multiply-add per tap
    flops = 5.0 * nt * math.log2(math.prod(n)) + 4.0 * M * taps + 2.0 * Nt
    one = 8 * d * M + c * (M + Nt)
    if case["kind"] == "step":
        return dict(bytes=8 * d * M + 2 * c * (M + Nt), flops=2 * flops)
    if case["kind"] == "cg":
        return dict(bytes=21 * one, flops=21 * flops)
    if case["kind"] == "autograd":
        return dict(bytes=2 * one + 16 * d * M + c * M, flops=2 * flops + 5.0 * nt * math.log2(math.prod(n)) + 4.0 * d * M * taps)
    return dict(bytes=2 * one, flops=2 * flops)


# ---------------------------------------------------------------- the same sums in 64 bits
class _Exact:
    """Windowed forward, adjoint and node gradient of one instance, torch float64 on the GPU."""

    def __init__(self, N, n, m, window, x):
        self.N, self.n, self.m, self.es = N, n, m, window == "es"
        self.d, self.W, self.x = len(N), 2 * m + 2, x
        self.sig = [b / a for a, b in zip(N, n)]
        self.b = [2 * s / (2 * s - 1) * m / math.pi for s in self.sig]
        self.alpha = m + 0.5
        self.beta = [0.97 * math.pi * 2 * self.alpha * (1 - 1 / (2 * s)) for s in self.sig]
        self.norm = 1.0 if self.es else math.prod(math.sqrt((2 * s - 1) / (2 * s * m)) for s in self.sig)
        self.roll = torch.ones([1] * self.d, dtype=torch.float64, device=DEV)
        for t in range(self.d):
            k = np.arange(N[t], dtype=np.float64) - N[t] // 2
            if self.es:
                z, w = np.polynomial.legendre.leggauss(96)
                y = 0.5 * self.alpha * (z + 1)
                phi = np.exp(self.beta[t] * (np.sqrt(1 - (y / self.alpha) ** 2) - 1))
                r = 1 / ((self.alpha * w * phi) @ np.cos(2 * np.pi * y[:, None] * k / n[t]))
            else:
                r = np.exp(math.pi ** 2 * self.b[t] / n[t] ** 2 * k * k)
            self.roll = self.roll * torch.from_numpy(r).to(DEV).reshape([-1 if i == t else 1 for i in range(self.d)])
        self.place = torch.meshgrid(*[torch.remainder(torch.arange(a, device=DEV) - a // 2, b) for a, b in zip(N, n)],
                                    indexing="ij")
        self.step = max(1, (1 << 25) // self.W ** self.d)

    def taps(self, x, deriv=False):
        """Grid indices and weights per dimension; with ``deriv`` their derivatives by x as well."""
        idx, w, dw = [], [], []
        l = torch.arange(self.W, device=DEV)
        for t in range(self.d):
            nx = x[:, t] * self.n[t]
            u = torch.round(nx).long() - torch.signbit(x[:, t]).long() - self.m
            y = (nx - u.double())[:, None] - l.double()
            if self.es:
                q = (1 - (y / self.alpha) ** 2).clamp_min(0)
                e = torch.where(q > 0, torch.exp(self.beta[t] * (q.sqrt() - 1)), torch.zeros_like(q))
                de = torch.where(q > 0, -e * self.beta[t] * y / (self.alpha ** 2 * q.sqrt().clamp_min(1e-300)), e)
            else:
                e = torch.exp(-y * y / self.b[t])
                de = -2 * y / self.b[t] * e
            idx.append(torch.remainder(u[:, None] + l, self.n[t]))
            w.append(e)
            dw.append(de * self.n[t])
        flat = idx[0]
        for t in range(1, self.d):
            flat = (flat[..., None] * self.n[t]) + idx[t].reshape([-1] + [1] * t + [self.W])
        return (flat, w, dw) if deriv else (flat, w)

    def grid(self, fh):
        g = torch.zeros(self.n, dtype=torch.complex128, device=DEV)
        g[self.place] = fh.to(torch.complex128) * self.roll
        return torch.fft.fftn(g).reshape(-1)

    def sum(self, v, w):
        for t in range(self.d - 1, -1, -1):
            v = (v * w[t].reshape([-1] + [1] * t + [self.W])).sum(-1)
        return v * self.norm

    def forward(self, fh):
        g, out = self.grid(fh), []
        for x in self.x.split(self.step):
            flat, w = self.taps(x)
            out.append(self.sum(g[flat], w))
        return torch.cat(out)

    def adjoint(self, f):
        g = torch.zeros(math.prod(self.n), 2, dtype=torch.float64, device=DEV)
        f = f.to(torch.complex128) * self.norm
        for x, v in zip(self.x.split(self.step), f.split(self.step)):
            flat, w = self.taps(x)
            for t in range(self.d):
                v = v[..., None] * w[t].reshape([-1] + [1] * t + [self.W])
            g.index_add_(0, flat.reshape(-1), torch.view_as_real(v.reshape(-1)))
        g = torch.view_as_complex(g).reshape(self.n)
        return (torch.fft.ifftn(g) * math.prod(self.n))[self.place] * self.roll

    def gradient(self, fh, gf):
        g, out = self.grid(fh), []
        for x, v in zip(self.x.split(self.step), gf.split(self.step)):
            flat, w, dw = self.taps(x, True)
            a = g[flat]
            out.append(torch.stack([(v.conj() * self.sum(a, w[:t] + [dw[t]] + w[t + 1:])).real for t in range(self.d)], 1))
        return torch.cat(out)


def _exact_ndft(N, x, fh, f):
    e = [torch.exp(-2j * math.pi * torch.remainder(x[:, t, None] * (torch.arange(N[t], device=DEV) - N[t] // 2), 1.0))
         for t in range(len(N))]
    fwd, rows = [], max(1, (1 << 25) // math.prod(N[:-1]))
    fh2 = fh.reshape(-1, N[-1])
    for lo in range(0, x.shape[0], rows):
        v = e[-1][lo:lo + rows] @ fh2.T
        for t in range(len(N) - 2, -1, -1):
            v = (v.reshape(v.shape[0], -1, N[t]) * e[t][lo:lo + rows, None, :]).sum(-1)
        fwd.append(v.reshape(-1))
    out = torch.zeros(math.prod(N[:-1]), N[-1], dtype=torch.complex128, device=DEV)
    for lo in range(0, x.shape[0], rows):
        v = f[lo:lo + rows, None]
        for t in range(len(N) - 1):
            v = (v[:, :, None] * e[t][lo:lo + rows, None, :].conj()).reshape(v.shape[0], -1)
        out += v.T @ e[-1][lo:lo + rows].conj()
    return [torch.cat(fwd), out.reshape(N)]


def exact(case, seed):
    N, n = _sizes(case)
    x, counts, fh, f = _inputs(case, seed)
    if case["kind"] == "ndft":
        return _exact_ndft(N, x, fh, f)
    if case["kind"] in ("step", "graph"):
        fwd, adj, lo = [], [], 0
        for i, M in enumerate(counts):
            E = _Exact(N, n, case["m"], case["window"], x[lo:lo + M])
            fwd.append(E.forward(fh[i] if case["batch"] > 1 else fh))
            adj.append(E.adjoint(f[lo:lo + M]))
            lo += M
        both = [torch.cat(fwd), torch.stack(adj) if case["batch"] > 1 else adj[0]]
        return both if case["kind"] == "step" else both[::-1]
    E = _Exact(N, n, case["m"], case["window"], x)
    if case["kind"] == "dropin":
        v = E.forward(fh)
        return [v.cpu().numpy(), E.adjoint(v).reshape(-1).cpu().numpy()]
    if case["kind"] == "autograd":
        y = E.forward(fh)
        r = 2 * (y - f)
        return [y, E.gradient(fh, r), E.adjoint(r)]
    # cg: x_{k+1} from x_0 = 0, ten iterations of conjugate gradients on A^H A x = A^H f
    v = torch.zeros(N, dtype=torch.complex128, device=DEV)
    r = E.adjoint(f)
    p, rr = r.clone(), torch.vdot(r.reshape(-1), r.reshape(-1)).real
    for _ in range(10):
        q = E.adjoint(E.forward(p))
        a = rr / torch.vdot(p.reshape(-1), q.reshape(-1)).real
        v, r = v + a * p, r - a * q
        new = torch.vdot(r.reshape(-1), r.reshape(-1)).real
        p, rr = r + new / rr * p, new
    return v
