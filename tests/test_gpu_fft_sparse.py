"""The fixed-point FFT of few large values among zeros or small ones, which do not grow as a dense
line's do: single coefficients against their exponential, and a large one beside small ones.

Tolerance: the exponential's, the ratio's and the result's roundings, 2^-53 each and once more."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

TOL = 4 * 2.0 ** -53


def _wave(n, k):
    t = [np.exp(-2j * np.pi * (((np.arange(a) * b) % a) / a)) for a, b in zip(n, k)]
    out = t[0]
    for v in t[1:]:
        out = out[..., None] * v
    return out


@pytest.mark.parametrize("N,n", [([20], [64]), ([100], [128]), ([500], [1024]), ([1000], [2048]), ([1500], [4096]), ([3000], [8192]), ([100000], None),
                                 ([16, 1200], [32, 4096]), ([400, 30], None), ([30, 60, 20], None)])
@pytest.mark.parametrize("where", ["first", "middle", "last"])
def test_single_coefficient(N, n, where):
    from cunfft_gb300.nfft import NFFT
    dev = torch.device("cuda:0")
    p = NFFT(N, n=n, m=2, precision="f64", device=dev).set_nodes(torch.zeros(1, len(N), dtype=torch.float64, device=dev))
    at = [{"first": 0, "middle": (2 * v) // 3, "last": v - 1}[where] for v in N]
    fh = torch.zeros(N, dtype=torch.complex128, device=dev)
    fh[tuple(at)] = 1.0  # a real factor times the wave
    p.forward(fh)
    g = p.grid().cpu().numpy()
    c = g.reshape(-1)[0].real
    d = g / c - _wave(p.n, [a - v // 2 for a, v in zip(at, N)])
    assert np.sqrt(np.mean(np.abs(d) ** 2)) < TOL * (1 + 0.5 * (len(N) - 1))  # the reference's products
    p.close()


@pytest.mark.parametrize("N", [[500], [1500], [40, 600]])
def test_large_value_beside_small_ones(N):
    """The transform of a sum is the sum of the transforms."""
    from cunfft_gb300.nfft import NFFT
    dev = torch.device("cuda:0")
    rng = np.random.default_rng(3)
    p = NFFT(N, m=2, precision="f64", device=dev).set_nodes(torch.zeros(1, len(N), dtype=torch.float64, device=dev))
    fh = torch.from_numpy(rng.uniform(-1, 1, N) + 1j * rng.uniform(-1, 1, N)).to(dev) * 1e-5
    fh.reshape(-1)[fh.numel() // 2 + 3] = 1.0 - 0.5j
    p.forward(fh)
    full = p.grid().clone()
    one = torch.zeros_like(fh)
    one.reshape(-1)[fh.numel() // 2 + 3] = 1.0 - 0.5j
    p.forward(fh - one)
    rest = p.grid().clone()
    p.forward(one)
    d = full - rest - p.grid()
    assert torch.linalg.norm(d) < 2 * TOL * torch.linalg.norm(full)
    p.close()
