"""3D FP32 spreading, the order in which CTAs take work items: fewer items than CTAs, whole
and partial rounds, wrapped tiles.  Against the FP64 plan.  Tolerance: FP16 hi/lo products
(3 2^-22) and FP32 taps (exponents below 45, one ulp each), together below 2e-6."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N,M", [([16, 16, 16], 1), ([16, 16, 16], 400), ([48, 40, 56], 100), ([48, 40, 56], 3000),
                                 ([64, 64, 64], 20000)])
def test_every_item_once(N, M):
    from cunfft_gb300.nfft import NFFT
    dev = torch.device("cuda:0")
    rng = np.random.default_rng(M)
    x = torch.from_numpy(rng.uniform(-0.5, 0.5, (M, 3))).to(dev)
    f = torch.from_numpy((rng.uniform(-1, 1, M) + 1j * rng.uniform(-1, 1, M)).astype(np.complex64)).to(dev)
    p = NFFT(N, m=6, precision="f32", device=dev).set_nodes(x)
    q = NFFT(N, m=6, precision="f64", device=dev).set_nodes(x)
    assert p.spread_kernel() == "tensor"
    g = p.spread(f).to(torch.complex128)
    ref = q.spread(f.to(torch.complex128))
    p.synchronize()
    q.synchronize()
    assert float(torch.linalg.norm(g - ref) / torch.linalg.norm(ref)) < 2e-6
    p.close()
    q.close()
