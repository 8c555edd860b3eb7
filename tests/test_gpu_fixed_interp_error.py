"""Interpolation error of the FP64 form's forward transform in 3D with wide windows: the window's
sum over the plan's own grid against extended-precision sums with exact taps.

Bound: the grid is what a low-pass window sums, its values cancel about (1 + m / 6)^3 times (24 at
m = 12); with sums of FP64 taps from the window's recurrence that left 1.2e-14 at m = 12, which the
fixed-point kernel (a tile's values cut to 2^-54 of their largest) has to stay below."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N,m,tol", [([24, 20, 22], 6, 2e-15), ([32, 32, 32], 8, 3e-15), ([32, 32, 32], 12, 1.2e-14), ([20, 24, 20], 12, 1.2e-14)])
def test_wide_windows(N, m, tol):
    from cunfft_gb300.nfft import NFFT
    dev = torch.device("cuda:0")
    rng = np.random.default_rng(m)
    M, W = 150, 2 * m + 2
    x = rng.uniform(-0.5, 0.5, (M, 3))
    fh = rng.uniform(-1, 1, N) + 1j * rng.uniform(-1, 1, N)
    p = NFFT(N, m=m, precision="f64", device=dev).set_nodes(torch.from_numpy(x).to(dev))
    got = p.forward(torch.from_numpy(fh).to(dev)).cpu().numpy()
    g = p.grid().cpu().numpy()
    norm, idx, w = 1.0, [], []
    for t in range(3):
        s = p.n[t] / N[t]
        b = np.longdouble(2 * s / (2 * s - 1) * m / np.pi)
        norm *= np.sqrt((2 * s - 1) / (2 * s * m))
        nx = x[:, t] * p.n[t]
        u = np.rint(nx).astype(int) - np.signbit(x[:, t]) - m
        y = (nx - u)[:, None].astype(np.longdouble) - np.arange(W)
        idx.append((u[:, None] + np.arange(W)) % p.n[t])
        w.append(np.exp(-y * y / b))
    ref = np.empty(M, dtype=complex)
    for j in range(M):
        v = g[np.ix_(idx[0][j], idx[1][j], idx[2][j])].astype(np.clongdouble)
        for t in range(3):
            v = (v * w[t][j].reshape([-1] + [1] * (2 - t))).sum(0)
        ref[j] = complex(v) * norm
    assert np.linalg.norm(got - ref) < tol * np.linalg.norm(ref)
    p.close()
