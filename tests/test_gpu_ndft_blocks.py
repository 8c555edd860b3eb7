"""The direct NDFT kernels against the oracle where their blocks of coefficients, row groups
and node stages begin and end, and on batched instances.

Tolerance: the oracle evaluates each phase from k x rounded to FP64, 2 pi 2^-53 |k x| per
term, below 4e-13 for |k x| <= 500 (N = 1000)."""
import numpy as np
import pytest

import oracle as O

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

TOL = 1e-12


def _rand(shape, rng):
    return rng.uniform(-1, 1, shape) + 1j * rng.uniform(-1, 1, shape)


@pytest.mark.parametrize("N", [[1], [2], [63], [64], [65], [130], [1000], [1, 64], [7, 65], [8, 63], [33, 129], [2, 3, 5],
                               [5, 9, 66], [3, 33, 4]])
@pytest.mark.parametrize("M", [1, 31, 33, 700])
def test_ndft_block_edges(N, M):
    from cunfft_gb300.nfft import NFFT
    dev = torch.device("cuda:0")
    rng = np.random.default_rng(M + sum(N))
    x, fh, f = rng.uniform(-0.5, 0.5, (M, len(N))), _rand(N, rng), _rand(M, rng)
    x[0] = -0.5
    p = NFFT(N, m=2, precision="f64", device=dev).set_nodes(torch.from_numpy(x).to(dev))
    assert O.rel_l2(O.ndft_forward(x, fh, N), p.ndft_forward(torch.from_numpy(fh).to(dev)).cpu().numpy()) < TOL
    got = p.ndft_adjoint(torch.from_numpy(f).to(dev)).cpu().numpy()
    assert O.rel_l2(O.ndft_adjoint(x, f, N).reshape(got.shape), got) < TOL
    p.close()


def test_ndft_batched_uneven():
    from cunfft_gb300.nfft import NFFT
    dev = torch.device("cuda:0")
    rng = np.random.default_rng(5)
    N, Ms = [10, 70], [0, 1, 300, 45]
    xs, fhs, fs = [rng.uniform(-0.5, 0.5, (M, 2)) for M in Ms], _rand([4] + N, rng), [_rand(M, rng) for M in Ms]
    p = NFFT(N, m=2, precision="f64", batch=4, device=dev).set_nodes(torch.from_numpy(np.concatenate(xs)).to(dev), Ms)
    fwd = p.ndft_forward(torch.from_numpy(fhs).to(dev)).cpu().numpy()
    adj = p.ndft_adjoint(torch.from_numpy(np.concatenate(fs)).to(dev)).cpu().numpy()
    lo = 0
    for i, M in enumerate(Ms):
        if M:
            assert O.rel_l2(O.ndft_forward(xs[i], fhs[i], N), fwd[lo:lo + M]) < TOL
            assert O.rel_l2(O.ndft_adjoint(xs[i], fs[i], N).reshape(N), adj[i]) < TOL
        else:
            assert not adj[i].any()
        lo += M
    p.close()
