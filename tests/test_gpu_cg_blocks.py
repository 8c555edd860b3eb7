"""Conjugate gradients take any number of iterations: the scalars are kept for a block at a time,
and blocks agree with one another.  Tolerance: as in test_gpu_cg_kernels.py."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def _case(M=400, N=(12, 10)):
    from cunfft_gb300.nfft import NFFT
    dev = torch.device("cuda:0")
    rng = np.random.default_rng(2)
    x = torch.from_numpy(rng.uniform(-0.5, 0.5, (M, len(N)))).to(dev)
    f = torch.from_numpy(rng.uniform(-1, 1, M) + 1j * rng.uniform(-1, 1, M)).to(dev)
    return NFFT(list(N), m=5, precision="f64", device=dev).set_nodes(x), f


def test_iterations_without_end_stop_at_the_tolerance():
    from cunfft_gb300.solver import cgne
    plan, f = _case()
    x, hist = cgne(plan, f, iters=10 ** 12, tol=1e-6, lam=1.0)
    ref, h2 = cgne(plan, f, iters=100, tol=1e-6, lam=1.0)
    assert len(hist) == len(h2) and hist[-1] <= 1e-6 < hist[-2]
    assert torch.linalg.norm(x - ref) < 1e-12 * torch.linalg.norm(ref)
    plan.close()


@pytest.mark.parametrize("callback", [False, True])
def test_blocks_agree(monkeypatch, callback):
    from cunfft_gb300 import solver
    plan, f = _case()
    ref, href = solver.cgne(plan, f, iters=11, lam=0.5)
    monkeypatch.setattr(solver, "_BLOCK", 4)
    seen = []
    got, hist = solver.cgne(plan, f, iters=11, lam=0.5, callback=(lambda v, r: seen.append(r)) if callback else None)
    assert len(hist) == 11 and np.allclose(hist, href, rtol=1e-2, atol=1e-12) and (not callback or seen == hist)
    assert torch.linalg.norm(got - ref) < 1e-12 * torch.linalg.norm(ref)
    plan.close()


def test_samples_of_other_shapes_and_strides():
    from cunfft_gb300.solver import cgne
    plan, f = _case()
    t = f.reshape(20, 20).t()
    ref, _ = cgne(plan, t.contiguous().reshape(-1), iters=5)
    got, _ = cgne(plan, t, iters=5)
    assert torch.linalg.norm(got - ref) < 1e-12 * torch.linalg.norm(ref)
    plan.close()


def test_negative_tolerance_never_stops():
    """As the recurrences themselves: a zero residual divides by zero in the next iteration."""
    from cunfft_gb300.nfft import NFFT
    from cunfft_gb300.solver import cgne
    dev = torch.device("cuda:0")
    plan = NFFT([1], m=6, precision="f64", device=dev).set_nodes(torch.zeros(1, 1, dtype=torch.float64, device=dev))
    f = torch.ones(1, dtype=torch.complex128, device=dev)
    _, h0 = cgne(plan, f, iters=6)
    _, h1 = cgne(plan, f, iters=6, tol=-1.0)
    assert len(h1) == 6 and h1[:len(h0)] == pytest.approx(h0, abs=1e-12)
    plan.close()
