"""The precision of the FP64 form's spreading does not hang on the scheduling option ``chunk``.

Tolerance: items of at most 512 nodes round every contribution to 2^-53 of their largest sample,
0.3 units each against a weight of some 0.2 on average, 1e-15 of a cell; the roll-off raises that
at most twofold per dimension at m = 6.  Two such results are compared."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N,T", [([200], 0), ([200], 64), ([40, 30], 0), ([12, 10, 14], 0)])
def test_large_chunks_keep_the_bits(N, T):
    from cunfft_gb300.nfft import NFFT
    dev = torch.device("cuda:0")
    rng = np.random.default_rng(len(N))
    M = 1 << 18
    x = torch.from_numpy(rng.uniform(0.0, 0.1, (M, len(N)))).to(dev)
    f = torch.from_numpy(rng.uniform(-1, 1, M) + 1j * rng.uniform(-1, 1, M)).to(dev)
    p = NFFT(N, m=6, precision="f64", device=dev).set_nodes(x)
    p.set_tiling([T] if T else None, 64)
    ref = p.adjoint(f).clone()
    p.set_tiling([T] if T else None, 1 << 20)
    assert p.tiling()["chunk"] == 1 << 20
    got = p.adjoint(f)
    assert torch.linalg.norm(got - ref) < 2e-15 * 2 ** len(N) * torch.linalg.norm(ref)
    p.close()
