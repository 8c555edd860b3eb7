"""Inverse NFFT: reconstruct Fourier coefficients from nonuniform samples.

The reference's README promises "the nonequispaced fast Fourier transform and
its inversion" (README:1) but ships no solver.  This module adds one as a caller
of the GB300 forward/adjoint pair: conjugate gradients on the normal equations
of the first kind,

    min_fhat || W^(1/2) (A fhat - f) ||_2^2 + lam ||fhat||_2^2
    (A^H W A + lam I) fhat = A^H W f,

with optional sample weights W (e.g. density compensation) and Tikhonov term
lam.  Every iteration costs one forward and one adjoint NFFT on the plan's
nodes; the vector algebra is three kernels on the same stream with their scalars on the
device, so the host waits once at the end and every 1024 iterations (every iteration with a callback
or a tolerance).
"""
import torch

from . import _native as nat
from .nfft import _ptr

_BLOCK = 1024  # iterations whose scalars are kept at a time


def cgne(plan, f, iters=20, weights=None, lam=0.0, fhat0=None, tol=0.0, callback=None):
    """Solve (A^H W A + lam I) fhat = A^H W f by conjugate gradients.

    plan: an ``NFFT`` with nodes bound; f: samples (M,) of the plan's dtype;
    weights: optional nonnegative (M,) real weights; returns (fhat, history),
    history the relative residual ||A^H W (f - A fhat) - lam fhat|| / ||A^H W f||
    per iteration.
    """
    cd = plan.cdtype
    f = f.to(cd)
    w = None if weights is None else weights.to(f.real.dtype)
    shape = plan._coef_shape()
    iters = int(iters)

    def normal_op(v, out=None, samples=None):
        av = plan.forward(v, out=samples)
        return plan.adjoint(av * w if w is not None else av, out=out)

    b = plan.adjoint(f * w if w is not None else f)
    x = torch.zeros(shape, dtype=cd, device=f.device) if fhat0 is None else fhat0.to(cd).clone().contiguous()
    r = b.clone()
    if fhat0 is not None:
        r -= normal_op(x)
        if lam:
            r -= lam * x
    if iters < 1:
        return x, []
    p, ap = r.clone(), torch.empty_like(r)
    samples = torch.empty(plan.M, dtype=cd, device=f.device)
    wait = callback is not None or tol > 0.0
    hist, scal, stop = [], None, None
    while len(hist) < iters:
        # every scalar stays on the device: <b, b>, <r, r> and <p, ap> per iteration, the history;
        # for a block of iterations, whose first <r, r> and flag are the last block's last
        n = min(iters - len(hist), _BLOCK)
        last, scal = scal, torch.zeros(2 + 3 * n, dtype=torch.float64, device=f.device)
        flag, stop = stop, torch.zeros(n + 1, dtype=torch.int32, device=f.device)
        args = [_ptr(t) for t in (b, x, r, p, ap, scal, stop)]

        def stage(kind, it):
            nat.check(plan._lib.cunfft_x_cg(plan._h, kind, it, n, float(lam), float(tol), *args), plan._h)

        if last is None:
            stage(0, 0)
        else:
            scal[0], scal[1], stop[0] = last[0], last[1 + _BLOCK], flag[_BLOCK]
        for it in range(n):
            normal_op(p, out=ap, samples=samples)
            stage(1, it)
            stage(2, it)
            stage(3, it)
            if wait:
                rel = scal[2 + 2 * n + it].item()
                hist.append(rel)
                if callback is not None:
                    callback(x.clone(), rel)
                if rel <= tol:
                    return x, hist
        if not wait:
            hist += scal[2 + 2 * n:].tolist()
            if tol >= 0.0 and 0.0 in hist:  # solved exactly: the iterations after it changed nothing
                del hist[hist.index(0.0) + 1:]
                break
    return x, hist
