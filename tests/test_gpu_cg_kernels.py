"""The conjugate-gradient kernels against the same recurrences in torch on the plan's own
transforms: sizes below and past one CTA, both precisions, weights, Tikhonov term, start
vector, batch; the waiting and the free-running loop agree.  Tolerance: the recurrences
magnify the transforms' run-to-run rounding (order of additions) by the condition number,
below 100 here."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def _plain(plan, f, iters, w, lam, x0):
    def op(v):
        av = plan.forward(v)
        return plan.adjoint(av * w if w is not None else av) + lam * v
    b = plan.adjoint(f * w if w is not None else f)
    x = torch.zeros_like(b) if x0 is None else x0.clone()
    r = b - op(x)
    p, hist = r.clone(), []
    dot = lambda a, c: torch.vdot(a.reshape(-1).to(torch.complex128), c.reshape(-1).to(torch.complex128)).real
    for _ in range(iters):
        ap, rr = op(p), dot(r, r)
        al = (rr / dot(p, ap)).to(f.real.dtype)
        x, r = x + al * p, r - al * ap
        new = dot(r, r)
        hist.append((new.sqrt() / dot(b, b).sqrt()).item())
        p = r + (new / rr).to(f.real.dtype) * p
    return x, hist


@pytest.mark.parametrize("prec,tol", [("f32", 2e-5), ("f64", 1e-12)])
@pytest.mark.parametrize("N,batch,extra", [([7], 1, ""), ([16], 1, "lam"), ([40, 33], 1, "w"), ([40, 33], 1, "x0 lam w"), ([12, 10], 3, "w")])
def test_cgne_matches_plain_recurrences(N, batch, extra, prec, tol):
    from cunfft_gb300.nfft import NFFT
    from cunfft_gb300.solver import cgne
    dev = torch.device("cuda:0")
    rng = np.random.default_rng(len(N) + batch)
    Ms = [5 * int(np.prod(N)) + i for i in range(batch)]
    M = sum(Ms)
    cd = torch.complex64 if prec == "f32" else torch.complex128
    x = torch.from_numpy(rng.uniform(-0.5, 0.5, (M, len(N)))).to(dev)
    rand = lambda shape: torch.from_numpy(rng.uniform(-1, 1, shape) + 1j * rng.uniform(-1, 1, shape)).to(dev, cd)
    f = rand(M)
    w = torch.from_numpy(rng.uniform(0.5, 2, M)).to(dev, f.real.dtype) if "w" in extra else None
    lam = 3.0 if "lam" in extra else 0.0
    plan = NFFT(N, m=5, precision=prec, batch=batch, device=dev).set_nodes(x, Ms)
    x0 = rand(plan._coef_shape()) if "x0" in extra else None
    ref, href = _plain(plan, f, 6, w, lam, x0)
    got, hist = cgne(plan, f, iters=6, weights=w, lam=lam, fhat0=x0)
    assert torch.linalg.norm(got - ref) < tol * torch.linalg.norm(ref) and np.allclose(hist, href, rtol=1e-2, atol=tol)
    seen = []
    again, h2 = cgne(plan, f, iters=6, weights=w, lam=lam, fhat0=x0, tol=href[3], callback=lambda v, rel: seen.append((v, rel)))
    assert len(h2) in (4, 5) and len(seen) == len(h2) and [s[1] for s in seen] == h2
    assert torch.equal(seen[-1][0], again) and not torch.equal(seen[0][0], again)
    plan.close()


def test_cgne_no_iterations_and_exact_solution():
    from cunfft_gb300.nfft import NFFT
    from cunfft_gb300.solver import cgne
    dev = torch.device("cuda:0")
    x = torch.linspace(-0.5, 0.49, 40, dtype=torch.float64, device=dev)[:, None]
    plan = NFFT([8], m=6, precision="f64", device=dev).set_nodes(x)
    f = torch.ones(40, dtype=torch.complex128, device=dev)
    sol, hist = cgne(plan, f, iters=0)
    assert hist == [] and not sol.any()
    sol, hist = cgne(plan, torch.zeros_like(f), iters=3)  # <b, b> = 0: not a number, as the plain recurrences
    assert len(hist) == 3 and np.isnan(hist).all()
    plan.close()
