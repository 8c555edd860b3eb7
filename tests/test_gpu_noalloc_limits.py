"""cunfft_x_spread_noalloc at its tile limit: 2D FP64 grids of 65536 tiles of 32 x 64 are accepted
(the plans' own tiles are 16 x 64) and right, larger ones are refused.

Tolerance: sums of 200 taps of a few 2^-53 each, 1e-14."""
import ctypes

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def _call(N, n, M, x, f, g, m=6):
    from cunfft_gb300 import _native as nat
    fn = nat.lib().cunfft_x_spread_noalloc
    vp = lambda t: ctypes.c_void_p(t if isinstance(t, int) else t.data_ptr())
    arr = lambda v: (ctypes.c_int64 * len(v))(*v)
    stream = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    return fn(len(N), arr(N), arr(n), m, nat.F64, ctypes.c_int64(M), vp(x), vp(f), vp(g), stream, None)


@pytest.mark.parametrize("N,n", [([8000, 4000], [16384, 8192]), ([5000, 5000], [10000, 10000])])
def test_2d_fp64_grids_at_the_limit(N, n):
    from cunfft_gb300 import _native as nat
    dev, m = torch.device("cuda:0"), 6
    x = np.array([[0.31, -0.27], [-0.5, 0.499999], [-0.0, 0.1], [0.31 + 20.3 / n[0], -0.27 + 3.1 / n[1]]])
    f = np.array([1 + 2j, 3 - 1j, -2j, 0.5])
    g = torch.zeros(n, dtype=torch.complex128, device=dev)
    assert _call(N, n, 4, torch.from_numpy(x).to(dev), torch.from_numpy(f).to(dev), g) == nat.SUCCESS
    torch.cuda.synchronize()
    ref, l = {}, np.arange(2 * m + 2)
    for j in range(4):
        w, idx, norm = [], [], 1.0
        for t in range(2):
            s = n[t] / N[t]
            nx = x[j, t] * n[t]
            u = int(np.rint(nx)) - int(np.signbit(x[j, t])) - m
            w.append(np.exp(-((nx - u) - l) ** 2 / (2 * s / (2 * s - 1) * m / np.pi)))
            idx.append((u + l) % n[t])
            norm *= np.sqrt((2 * s - 1) / (2 * s * m))
        for a in l:
            for b in l:
                k = (int(idx[0][a]), int(idx[1][b]))
                ref[k] = ref.get(k, 0) + f[j] * norm * w[0][a] * w[1][b]
    at = torch.tensor(sorted(ref), device=dev)
    got, want = g[at[:, 0], at[:, 1]].cpu().numpy(), np.array([ref[k] for k in sorted(ref)])
    assert np.linalg.norm(got - want) < 1e-14 * np.linalg.norm(want)
    assert torch.count_nonzero(torch.view_as_real(g).abs().sum(-1)).item() <= len(ref)


def test_larger_grids_are_refused():
    from cunfft_gb300 import _native as nat
    assert _call([8000, 8000], [16384, 16384], 10, 1, 1, 1) == nat.INVALID_ARGUMENT
    assert _call([1 << 26], [1 << 27], 10, 1, 1, 1) == nat.INVALID_ARGUMENT
