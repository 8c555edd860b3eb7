"""Work items of the binning: tiles and sub-tiles with few and with very many items, side by
side and alone in their warp of 32.  Every node must be in one item of its own tile: the
transform agrees with the oracle, whole numbers of nodes per tile included."""
import numpy as np
import pytest

import oracle as O

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


# tolerance: FP32 sums of up to 20000 nodes on a cell, 2^-24 sqrt(20000) = 8.4e-6 at random signs
@pytest.mark.parametrize("prec,tol", [("f64", 1e-13), ("f32", 2e-5)])
@pytest.mark.parametrize("N,chunk", [([700], 0), ([64, 90], 0), ([64, 90], 33), ([33, 45], 0), ([20, 24, 28], 0), ([20, 24, 28], 32)])
def test_dense_and_sparse_tiles(N, chunk, prec, tol):
    from cunfft_gb300.nfft import NFFT
    dev = torch.device("cuda:0")
    rng = np.random.default_rng(len(N) * 10 + chunk)
    d = len(N)
    x = np.concatenate([rng.normal(0.1, 1e-4, (20000, d)), rng.normal(-0.3, 1e-3, (700, d)), rng.uniform(-0.5, 0.5, (900, d)),
                        np.full((5, d), 0.45)])
    x = x[rng.permutation(len(x))]
    f = rng.uniform(-1, 1, len(x)) + 1j * rng.uniform(-1, 1, len(x))
    p = NFFT(N, m=5, precision=prec, device=dev)
    if chunk:
        p.set_tiling(None, chunk)
    p.set_nodes(torch.from_numpy(x).to(dev))
    g = rng.uniform(-1, 1, p.n) + 1j * rng.uniform(-1, 1, p.n)
    got = p.spread(torch.from_numpy(f).to(dev)).cpu().numpy()
    assert O.rel_l2(O.spread(x, f, N, p.n, 5), got) < tol
    got = p.interp(torch.from_numpy(g).to(dev)).cpu().numpy()
    assert O.rel_l2(O.interp(x, g, N, p.n, 5), got) < tol
    p.close()
