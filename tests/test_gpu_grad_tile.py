"""The FP32 form's tiled node gradient against the FP64 form's one-thread-per-node kernel at
the edges of tiles, items and warp batches, every width class, both windows.  Tolerance: the
FP32 form's bar of the other kernels (FP32 FFT, taps and sums), 1e-5."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

TOL = 1e-5


@pytest.mark.parametrize("window", ["gaussian", "es"])
@pytest.mark.parametrize("N,n,m", [([90], None, 6), ([50], [101], 3), ([40, 70], None, 6), ([33, 31], [67, 71], 4), ([48, 40], None, 9),
                                   ([64, 64], None, 1), ([40, 36], None, 15), ([18, 20, 24], None, 6), ([11, 9, 13], [23, 19, 27], 3),
                                   ([12, 16, 14], None, 8), ([16, 16, 16], None, 14)])
@pytest.mark.parametrize("M", [1, 9, 2100])
def test_tiled_gradient_matches_fp64_kernel(N, n, m, window, M):
    from cunfft_gb300.nfft import NFFT
    dev = torch.device("cuda:0")
    rng = np.random.default_rng(M + m)
    d = len(N)
    x = rng.uniform(-0.5, 0.5, (M, d))
    x[M // 2:] *= 0.05  # several items in the centre tiles
    x[0] = -0.5
    x = torch.from_numpy(x).to(dev)
    fh = torch.from_numpy(rng.uniform(-1, 1, N) + 1j * rng.uniform(-1, 1, N)).to(dev)
    gf = torch.from_numpy(rng.uniform(-1, 1, M) + 1j * rng.uniform(-1, 1, M)).to(dev)
    got = {}
    for prec in ("f32", "f64"):
        p = NFFT(N, n=n, m=m, precision=prec, device=dev, window=window).set_nodes(x)
        got[prec] = p.node_gradient(fh, gf)
        p.close()
    assert torch.linalg.norm(got["f32"] - got["f64"]) < TOL * torch.linalg.norm(got["f64"])


def test_tiled_gradient_batched_and_non_finite_node():
    from cunfft_gb300.nfft import NFFT
    dev = torch.device("cuda:0")
    rng = np.random.default_rng(3)
    Ms = [0, 5, 700]
    x = torch.from_numpy(rng.uniform(-0.5, 0.5, (705, 2))).to(dev)
    x[9, 1] = float("nan")
    fh = torch.from_numpy(rng.uniform(-1, 1, (3, 20, 24)) + 0j).to(dev)
    gf = torch.from_numpy(rng.uniform(-1, 1, 705) + 1j).to(dev)
    got = [NFFT([20, 24], m=5, precision=q, batch=3, device=dev).set_nodes(x, Ms).node_gradient(fh, gf) for q in ("f32", "f64")]
    ok = torch.arange(705, device=dev) != 9
    assert torch.isnan(got[0][9]).all() and torch.isnan(got[1][9]).any()
    assert torch.linalg.norm(got[0][ok] - got[1][ok]) < TOL * torch.linalg.norm(got[1][ok])
