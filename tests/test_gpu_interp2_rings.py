"""2D FP32 interpolation, the rings of sub-tiles: item sizes that fill some of the four lane
quarters, item sequences longer than a loader's 32-item window, tiny and wrapped grids.
Against the FP64 plan's interpolation of the same grid.  Tolerance, of the sum of the taps
times |G|: FP16 hi/lo products (3 2^-22) and FP32 taps (exponents below 45, one ulp each),
together below 4e-6."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

TOL = 4e-6


def _check(N, m, x, n=None, window="gaussian"):
    from cunfft_gb300.nfft import NFFT
    dev = torch.device("cuda:0")
    xd = torch.from_numpy(x).to(dev)
    p = NFFT(N, n=n, m=m, precision="f32", device=dev, window=window).set_nodes(xd)
    q = NFFT(N, n=n, m=m, precision="f64", device=dev, window=window).set_nodes(xd)
    assert p.interp_kernel() == "tensor"
    gen = torch.Generator(device=dev).manual_seed(3)
    g = torch.view_as_complex(torch.randn(*p.n, 2, generator=gen, device=dev))
    f = p.interp(g)
    ref = q.interp(g.to(torch.complex128))
    mag = q.interp(g.to(torch.complex128).abs().to(torch.complex128)).real
    p.synchronize()
    q.synchronize()
    assert bool(((f.to(torch.complex128) - ref).abs() <= TOL * mag + 1e-30).all())
    p.close()
    q.close()


@pytest.mark.parametrize("window", ["gaussian", "es"])
@pytest.mark.parametrize("m", [1, 4, 7])
def test_widths(m, window):
    _check([64, 48], m, np.random.default_rng(m).uniform(-0.5, 0.5, (9000, 2)), window=window)


@pytest.mark.parametrize("counts", [(1,), (32, 33), (31, 96, 97, 1), (128, 129, 64, 65, 5, 300)])
def test_lane_quarters(counts):
    """counts[i] nodes in sub-tile i of a row of sub-tiles at the wrap."""
    rng = np.random.default_rng(len(counts))
    x = [np.stack([0.499 - rng.uniform(0, 0.02, c), -0.49 + 0.0625 * i + rng.uniform(0, 0.01, c)], 1)
         for i, c in enumerate(counts)]
    _check([128, 128], 6, np.concatenate(x))


@pytest.mark.parametrize("N,M", [([1024, 1024], 40000), ([2048, 2048], 70001)])
def test_long_item_sequences(N, M):
    _check(N, 3, np.random.default_rng(M).uniform(-0.5, 0.5, (M, 2)))


@pytest.mark.parametrize("N,n", [([4, 8], [8, 16]), ([10, 100], [20, 200]), ([9, 50], [19, 104])])
def test_small_grids(N, n):
    _check(N, 6, np.random.default_rng(n[0]).uniform(-0.5, 0.5, (500, 2)), n=n)
