"""The FP64 form's fixed-point FFT against torch's: line lengths 16 to 4096 (both parities of
log2), 1D in two passes, several dimensions, oversampling from none to eight-fold, batches,
extreme and non-finite values.  Tolerance: an FP64 FFT's own error, a few 2^-53 log2 n."""
import math

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

TOL = 1e-14


def _padded(p, fh):
    """Coefficients times the Gaussian roll-off factors on the zero-padded grid (one instance)."""
    g = torch.zeros(p.n, dtype=torch.complex128, device=fh.device)
    place = torch.meshgrid(*[torch.remainder(torch.arange(a, device=fh.device) - a // 2, b) for a, b in zip(p.N, p.n)], indexing="ij")
    v = fh.clone()
    for t, (a, b) in enumerate(zip(p.N, p.n)):
        s = b / a
        fac = math.pi ** 2 * (2 * s / (2 * s - 1) * p.m / math.pi) / b ** 2
        k = torch.arange(a, device=fh.device, dtype=torch.float64) - a // 2
        v = v * torch.exp(fac * k * k).reshape([-1 if i == t else 1 for i in range(p.d)])
    g[place] = v
    return g


def _rel(a, b):
    return (torch.linalg.norm(a - b) / torch.linalg.norm(b)).item()


@pytest.mark.parametrize("N,n,batch", [([8], [16], 1), ([16], [16], 3), ([9], [32], 1), ([100], [256], 2), ([200], [512], 1), ([512], [1024], 1),
                                       ([1000], [2048], 2), ([2048], [4096], 1), ([3001], [8192], 2), ([5000], [16384], 1), ([131072], None, 1),
                                       ([8, 8], None, 1), ([5, 16], [16, 16], 3), ([33, 100], [128, 256], 1), ([16, 1200], [32, 4096], 1),
                                       ([700, 20], [2048, 64], 1), ([8, 9, 10], [16, 32, 16], 2), ([16, 16, 16], [16, 16, 16], 1),
                                       ([20, 30, 40], [64, 64, 128], 1)])
def test_forward_and_adjoint_grids(N, n, batch):
    from cunfft_gb300.nfft import NFFT
    dev = torch.device("cuda:0")
    rng = np.random.default_rng(sum(N))
    M = 50
    x = torch.from_numpy(rng.uniform(-0.5, 0.5, (M * batch, len(N)))).to(dev)
    p = NFFT(N, n=n, m=2, precision="f64", batch=batch, device=dev).set_nodes(x, [M] * batch)
    rand = lambda s: torch.from_numpy(rng.uniform(-1, 1, s) + 1j * rng.uniform(-1, 1, s)).to(dev)
    fh, f = rand([batch] + N), rand(M * batch)
    p.forward(fh)
    got = p.grid().reshape([batch] + p.n)
    for i in range(batch):
        assert _rel(got[i], torch.fft.fftn(_padded(p, fh[i]))) < TOL
    g = p.spread(f).reshape([batch] + p.n)
    out = p.adjoint(f).reshape([batch] + N)
    got = p.grid().reshape([batch] + p.n)
    for i in range(batch):
        ref = torch.fft.ifftn(g[i]) * math.prod(p.n)
        assert _rel(got[i], ref) < TOL
        one = _padded(p, torch.ones(N, dtype=torch.complex128, device=dev))
        crop = (ref * one)[torch.meshgrid(*[torch.remainder(torch.arange(a, device=dev) - a // 2, b) for a, b in zip(p.N, p.n)],
                                          indexing="ij")]
        assert _rel(out[i], crop) < TOL
    p.close()


@pytest.mark.parametrize("scale", [1e-306, 1e-270, 1e270])
@pytest.mark.parametrize("N", [[100], [20, 24], [6000]])
def test_scales(N, scale):
    from cunfft_gb300.nfft import NFFT
    dev = torch.device("cuda:0")
    rng = np.random.default_rng(1)
    p = NFFT(N, m=2, precision="f64", device=dev).set_nodes(torch.zeros(1, len(N), dtype=torch.float64, device=dev))
    fh = torch.from_numpy(rng.uniform(-1, 1, N) + 1j * rng.uniform(-1, 1, N)).to(dev)
    p.forward(fh * scale)
    assert _rel(p.grid() / scale, torch.fft.fftn(_padded(p, fh))) < (TOL if scale > 1e-300 else 1e-12)
    p.forward(fh * 0)
    assert not p.grid().abs().any()
    p.close()


@pytest.mark.parametrize("bad", [float("nan"), float("inf")])
def test_non_finite_coefficient_spoils_the_whole_grid(bad):
    from cunfft_gb300.nfft import NFFT
    dev = torch.device("cuda:0")
    p = NFFT([16, 20], m=2, precision="f64", device=dev).set_nodes(torch.zeros(1, 2, dtype=torch.float64, device=dev))
    fh = torch.ones(16, 20, dtype=torch.complex128, device=dev)
    fh[3, 7] = bad
    assert not torch.isfinite(p.forward(fh)).any() and not torch.isfinite(p.grid()).any()
    p.close()
