"""FP32 shared-tile spreading in 1D and 2D, whose clusters of eight CTAs add the tiles of
neighbouring items: item counts around the cluster's, groups over several tiles and instances,
and the error on dense grids of few tiles.

Tolerances: against the oracle the FP32 form's bar of the other kernels; the dense grids' errors
against the FP64 form are those of items of 2048 nodes (2.1e-7, 5.0e-7, 2.8e-7), and a tenth for
the order of additions."""
import numpy as np
import pytest

import oracle as O

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N,n,m", [([16], None, 2), ([173], None, 4), ([90], [181], 3), ([3000], None, 6), ([2100], [4201], 9), ([20, 24], None, 9),
                                   ([40, 33], [81, 67], 10), ([64, 90], None, 15), ([30, 40], None, 4)])
@pytest.mark.parametrize("chunk,M", [(32, 1), (32, 31), (32, 33), (32, 255), (32, 257), (32, 3000), (0, 5000), (300, 5000)])
def test_against_the_oracle(N, n, m, chunk, M):
    from cunfft_gb300.nfft import NFFT
    dev = torch.device("cuda:0")
    rng = np.random.default_rng(M + m)
    x = rng.uniform(-0.5, 0.5, (M, len(N)))
    x[M // 2:] *= 0.02  # items of one tile beside items of many
    f = rng.uniform(-1, 1, M) + 1j * rng.uniform(-1, 1, M)
    p = NFFT(N, n=n, m=m, precision="f32", device=dev).set_nodes(torch.from_numpy(x).to(dev))
    p.set_spread_kernel("shared")
    p.set_tiling(None, chunk)
    for _ in range(2):
        got = p.spread(torch.from_numpy(f).to(dev)).cpu().numpy()
        assert O.rel_l2(O.spread(x, f, N, p.n, m), got) < 1e-5
    p.close()


def test_uneven_instances():
    from cunfft_gb300.nfft import NFFT
    dev = torch.device("cuda:0")
    rng = np.random.default_rng(9)
    N, Ms = [50], [700, 0, 1, 40, 3000]
    x = rng.uniform(-0.5, 0.5, (sum(Ms), 1))
    f = rng.uniform(-1, 1, sum(Ms)) + 1j * rng.uniform(-1, 1, sum(Ms))
    p = NFFT(N, m=5, precision="f32", batch=5, device=dev).set_nodes(torch.from_numpy(x).to(dev), Ms)
    got, lo = p.spread(torch.from_numpy(f).to(dev)).cpu().numpy(), 0
    for i, M in enumerate(Ms):
        if M:
            assert O.rel_l2(O.spread(x[lo:lo + M], f[lo:lo + M], N, p.n, 5), got[i]) < 1e-5
        else:
            assert not got[i].any()
        lo += M
    p.close()


@pytest.mark.parametrize("N,m,M,err", [([173], 4, 100000, 2.1e-7), ([30, 30], 9, 100000, 5.0e-7), ([2000], 6, 100000, 2.8e-7)])
def test_dense_grids_of_few_tiles(N, m, M, err):
    from cunfft_gb300.nfft import NFFT
    dev = torch.device("cuda:0")
    g = torch.Generator(device=dev).manual_seed(5)
    x = torch.rand(M, len(N), generator=g, device=dev, dtype=torch.float64) - 0.5
    f = torch.view_as_complex(torch.rand(M, 2, generator=g, device=dev, dtype=torch.float64) * 2 - 1).to(torch.complex64)
    out = []
    for prec in ("f32", "f64"):
        p = NFFT(N, m=m, precision=prec, device=dev).set_nodes(x)
        out.append(p.adjoint(f).to(torch.complex128))
        p.close()
    assert torch.linalg.norm(out[0] - out[1]) < 1.1 * err * torch.linalg.norm(out[1])
