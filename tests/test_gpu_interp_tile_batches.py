"""Shared-tile FP32 interpolation: a tile's nodes split into equal batches per warp, a lane
per tap, four nodes' sums reduced together."""
import numpy as np
import pytest
import torch

import oracle as O

pytestmark = pytest.mark.gpu

# Relative l2 error of the FP32 sums: three taps of 2^-22 (exp2) + 3 x 2^-24 (its argument, near
# the window's centre) each, and sums of at most 26 + 26 + 5 roundings of 2^-24 that add like a
# random walk, about 2^-21.2; doubled twice for the ES window's exponent and cancellation.
TOL = 2e-6


@pytest.mark.parametrize("N,n,m,window", [([30], [70], 6, "gaussian"), ([18, 20], [39, 45], 4, "es"),
                                          ([10, 12, 14], [21, 26, 29], 4, "es"), ([10, 12, 14], [22, 24, 33], 3, "gaussian"),
                                          ([20, 14, 16], [40, 32, 36], 8, "gaussian"),
                                          ([20, 16, 16], [42, 32, 36], 12, "gaussian")])
@pytest.mark.parametrize("count", [1, 7, 8, 9, 31, 33, 65, 270])
def test_one_tile_of_few_nodes(N, n, m, window, count):
    """Node counts around the multiples of the warps and of their batches, all in one tile
    (corner of the grid, windows wrapping)."""
    from cunfft_gb300.nfft import NFFT
    d = len(N)
    rng = np.random.default_rng(100 * d + count + m)
    x = -0.5 + rng.uniform(0, 1, (count, d)) * (3.0 / np.array(n))
    g = rng.uniform(-1, 1, n) + 1j * rng.uniform(-1, 1, n)
    p = NFFT(N, n=n, m=m, precision="f32", window=window, device="cuda:0").set_nodes(torch.from_numpy(x).to("cuda:0"))
    p.set_interp_kernel("shared")
    got = p.interp(torch.from_numpy(g).to("cuda:0", torch.complex64)).cpu().numpy()
    q = NFFT(N, n=n, m=m, precision="f64", window=window, device="cuda:0").set_nodes(torch.from_numpy(x).to("cuda:0"))
    ref = q.interp(torch.from_numpy(g).to("cuda:0")).cpu().numpy()
    if window == "gaussian":
        assert O.rel_l2(O.interp(x, g, N, n, m), ref) < 1e-12
    assert O.rel_l2(ref, got) < TOL
    p.close()
    q.close()
