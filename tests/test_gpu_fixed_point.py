"""The FP64 form's fixed-point gridding kernels against the oracle: every tap count class
(whole tiles and slabs of planes), tile and item edges, scales far from one, zero, infinite
and NaN values.

Tolerance: the oracle's taps come from the fast-Gaussian-gridding recurrence, whose W steps of
four roundings each leave up to 4 W 2^-53 per tap and dimension, 4e-14 for W = 32 in 3D; the
fixed-point kernels stay below that (2^-53 of the tile's largest value per node)."""
import numpy as np
import pytest

import oracle as O

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

TOL = 1e-13


@pytest.fixture(scope="module")
def dev():
    from cunfft_gb300 import _native
    _native.lib()
    return torch.device("cuda:0")


def _rand(shape, rng):
    return rng.uniform(-1, 1, shape) + 1j * rng.uniform(-1, 1, shape)


def _both(p, x, N, m, rng, dev, tol=TOL, window="gaussian", scale=1.0):
    g, f = _rand(p.n, rng) * scale, _rand(x.shape[0], rng) * scale
    got = p.interp(torch.from_numpy(g).to(dev)).cpu().numpy()
    assert O.rel_l2(O.interp(x, g, N, p.n, m, window=window) / scale, got / scale) < tol
    got = p.spread(torch.from_numpy(f).to(dev)).cpu().numpy()
    assert O.rel_l2(O.spread(x, f, N, p.n, m, window=window) / scale, got / scale) < tol


@pytest.mark.parametrize("window", ["gaussian", "es"])
@pytest.mark.parametrize("N,m", [([40], 1), ([700], 6), ([600], 15), ([33, 20], 2), ([64, 70], 6), ([40, 90], 7), ([50, 40], 12),
                                 ([40, 33], 15), ([12, 20, 18], 1), ([20, 12, 24], 4), ([24, 20, 33], 6), ([20, 18, 20], 7),
                                 ([18, 20, 22], 8), ([16, 20, 24], 12), ([16, 17, 20], 15)])
def test_every_width_class(dev, N, m, window):
    from cunfft_gb300.nfft import NFFT
    rng = np.random.default_rng(100 * len(N) + m)
    # 1537 nodes in one corner tile (several items) beside 2000 anywhere, and the box's edges
    x = np.concatenate([rng.uniform(0.0, 0.02, (1537, len(N))), rng.uniform(-0.5, 0.5, (2000, len(N)))])
    x[:3] = -0.5
    x[3:5] = np.nextafter(0.5, 0)
    x[5] = -0.0
    p = NFFT(N, m=m, precision="f64", device=dev, window=window).set_nodes(torch.from_numpy(x).to(dev))
    _both(p, x, N, m, rng, dev, window=window)
    p.close()


@pytest.mark.parametrize("N,n", [([9, 7, 11], [20, 15, 23]), ([5, 30, 6], [11, 61, 13]), ([31, 17], [63, 37]), ([37], [75])])
@pytest.mark.parametrize("M", [1, 2, 17, 511, 513])
def test_odd_grids_and_item_edges(dev, N, n, M):
    from cunfft_gb300.nfft import NFFT
    rng = np.random.default_rng(M + n[0])
    x = rng.uniform(-0.5, 0.5, (M, len(N)))
    p = NFFT(N, n=n, m=5, precision="f64", device=dev).set_nodes(torch.from_numpy(x).to(dev))
    _both(p, x, N, 5, rng, dev)
    p.set_tiling([2 if len(N) == 3 else 16], 64)
    _both(p, x, N, 5, rng, dev)
    p.close()


@pytest.mark.parametrize("N,m", [([64], 6), ([24, 30], 6), ([12, 14, 16], 6), ([12, 10, 14], 9)])
@pytest.mark.parametrize("scale", [1e-295, 1e-250, 1e250])
def test_scales_at_both_ends(dev, N, m, scale):
    """1e-295 and 1e250 take the FP64 items, 1e-250 the scaled integers."""
    from cunfft_gb300.nfft import NFFT
    rng = np.random.default_rng(7)
    x = rng.uniform(-0.5, 0.5, (900, len(N)))
    p = NFFT(N, m=m, precision="f64", device=dev).set_nodes(torch.from_numpy(x).to(dev))
    _both(p, x, N, m, rng, dev, scale=scale)
    p.close()


@pytest.mark.parametrize("N,m", [([400], 6), ([64, 64], 6), ([24, 24, 24], 6), ([24, 24, 24], 9)])
@pytest.mark.parametrize("bad", [np.nan, np.inf])
def test_zero_and_non_finite_values(dev, N, m, bad):
    from cunfft_gb300.nfft import NFFT
    rng = np.random.default_rng(11)
    d, M = len(N), 3000
    x = rng.uniform(-0.5, 0.5, (M, d))
    p = NFFT(N, m=m, precision="f64", device=dev).set_nodes(torch.from_numpy(x).to(dev))
    z = torch.zeros(p.n, dtype=torch.complex128, device=dev)
    assert not p.interp(z).abs().any() and not p.spread(torch.zeros(M, dtype=torch.complex128, device=dev)).abs().any()
    # one bad sample: its window's cells are not finite, the others are as without it
    f = _rand(M, rng)
    f0 = f.copy()
    f[5], f0[5] = bad, 0
    got, ref = p.spread(torch.from_numpy(f).to(dev)).cpu().numpy(), O.spread(x, f0, N, p.n, m)
    one = np.zeros(M, dtype=complex)
    one[5] = 1
    hit = O.spread(x, one, N, p.n, m) != 0
    assert not np.isfinite(got[hit]).any() and np.isfinite(got[~hit]).all()
    assert O.rel_l2(ref[~hit], got[~hit]) < TOL
    # one bad grid point: the nodes whose window holds it
    g = _rand(p.n, rng)
    at = tuple(v // 2 for v in p.n)
    g[at] = 0
    ref = O.interp(x, g, N, p.n, m)
    e = np.zeros(p.n, dtype=complex)
    e[at] = 1
    hit = O.interp(x, e, N, p.n, m) != 0
    g[at] = bad
    got = p.interp(torch.from_numpy(g).to(dev)).cpu().numpy()
    assert hit.any() and not np.isfinite(got[hit]).any() and np.isfinite(got[~hit]).all()
    assert O.rel_l2(ref[~hit], got[~hit]) < TOL
    p.close()
