"""2D FP32 spreading by sub-tiles against the oracle: item and operand-stage edges, every
width, both windows, wrapped and tiny grids, 8-byte aligned grids, sample scales, batches,
and the sparse grids that go to the whole-tile kernel.  Tolerance: FP16 hi/lo products
(3 2^-22) and FP32 taps (exponents below 45, one ulp each), together below 2e-6."""
import numpy as np
import pytest

import oracle as O

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

TOL = 2e-6


def _rand(n, rng):
    return rng.uniform(-1, 1, n) + 1j * rng.uniform(-1, 1, n)


def _check(N, m, x, rng, n=None, window="gaussian", scale=1.0, offset=0):
    from cunfft_gb300.nfft import NFFT
    dev = torch.device("cuda:0")
    p = NFFT(N, n=n, m=m, precision="f32", device=dev, window=window).set_nodes(torch.from_numpy(x).to(dev))
    assert p.spread_kernel() == "tensor"
    f = _rand(x.shape[0], rng).astype(np.complex64)
    buf = torch.zeros(int(np.prod(p.n)) + offset, dtype=torch.complex64, device=dev)
    g = p.spread(torch.from_numpy(f).to(dev) * scale, buf[offset:].reshape(p.n))
    p.synchronize()
    ref = O.spread(x, f.astype(np.complex128), N, p.n, m, window=window)
    assert O.rel_l2(ref, (g.cpu().numpy().astype(np.complex128) / scale)) < TOL
    p.close()


@pytest.mark.parametrize("window", ["gaussian", "es"])
@pytest.mark.parametrize("m", [1, 2, 3, 4, 5, 6, 7])
def test_every_width(m, window):
    rng = np.random.default_rng(m)
    _check([64, 48], m, rng.uniform(-0.5, 0.5, (9000, 2)), rng, window=window)


@pytest.mark.parametrize("count", [1, 15, 16, 17, 32, 33, 64, 65, 127, 128, 129, 300])
def test_item_and_stage_edges(count):
    """`count` nodes in one sub-tile at the wrap of both dimensions, one node elsewhere."""
    rng = np.random.default_rng(count)
    x = np.concatenate([0.499 + rng.uniform(-0.02, 0.0, (count, 2)), [[0.1, -0.2]]])
    _check([128, 128], 6, x, rng)


@pytest.mark.parametrize("N,n", [([4, 4], [8, 8]), ([4, 8], [8, 16]), ([8, 12], [16, 24]), ([10, 100], [20, 200]), ([30, 20], [61, 40]),
                                 ([9, 50], [19, 104])])
def test_small_and_odd_grids(N, n):
    rng = np.random.default_rng(n[0])
    _check(N, 6, rng.uniform(-0.5, 0.5, (500, 2)), rng, n=n)


@pytest.mark.parametrize("scale,offset", [(1.0, 1), (1e-30, 0), (1e30, 0), (3e-38, 0)])
def test_scales_and_alignment(scale, offset):
    rng = np.random.default_rng(5)
    _check([64, 64], 6, rng.uniform(-0.5, 0.5, (5000, 2)), rng, scale=scale, offset=offset)


@pytest.mark.parametrize("M", [3000, 12000, 40000])
def test_sparse_and_dense_sides_of_the_rule(M):
    rng = np.random.default_rng(M)
    _check([512, 512], 6, rng.uniform(-0.5, 0.5, (M, 2)), rng)


def test_batch_with_empty_and_zero_instances():
    from cunfft_gb300.nfft import NFFT
    dev = torch.device("cuda:0")
    rng = np.random.default_rng(9)
    N, Ms = [32, 40], [0, 700, 1, 260]
    xs = [rng.uniform(-0.5, 0.5, (M, 2)) for M in Ms]
    fs = [_rand(M, rng).astype(np.complex64) for M in Ms]
    fs[3] *= 0
    p = NFFT(N, m=5, precision="f32", batch=4, device=dev).set_nodes(torch.from_numpy(np.concatenate(xs)).to(dev), Ms)
    g = p.spread(torch.from_numpy(np.concatenate(fs)).to(dev)).cpu().numpy()
    p.synchronize()
    for i, M in enumerate(Ms):
        if M and i != 3:
            assert O.rel_l2(O.spread(xs[i], fs[i].astype(np.complex128), N, p.n, 5), g[i]) < TOL
        else:
            assert not g[i].any()
    p.close()
