"""Instances of a batched FP64 plan whose magnitudes differ do not see each other: neighbouring
lines of the fixed-point FFT belong to different instances wherever an instance's line count is
not a multiple of a CTA's lines.  Each instance against a plan of its own.

Tolerance: two FFTs' own errors, a few 2^-53 log2 n each, and two spreadings' of 2^-53 per cell."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

TOL = 1e-14
AMPS = [1.0, 1e-9, 0.0, 1e12, 1e-18, 1e-270, 1e-20]


@pytest.mark.parametrize("N,n", [([8], [16]), ([30], [64]), ([50], None), ([500], [1024]), ([700], [2048]), ([24, 20], None), ([5, 16], [16, 32]),
                                 ([50, 50], None), ([9, 10, 11], None), ([3, 20, 7], [16, 64, 16])])
def test_each_instance_as_alone(N, n):
    from cunfft_gb300.nfft import NFFT
    dev = torch.device("cuda:0")
    rng = np.random.default_rng(sum(N))
    B, M = len(AMPS), 40
    x = torch.from_numpy(rng.uniform(-0.5, 0.5, (B * M, len(N)))).to(dev)
    amp = torch.tensor(AMPS, dtype=torch.float64, device=dev)
    rand = lambda s: torch.from_numpy(rng.uniform(-1, 1, s) + 1j * rng.uniform(-1, 1, s)).to(dev)
    fh = rand([B] + N) * amp.reshape([B] + [1] * len(N))
    f = rand([B, M]) * amp[:, None]
    p = NFFT(N, n=n, m=3, precision="f64", batch=B, device=dev).set_nodes(x, [M] * B)
    fwd, adj = p.forward(fh).reshape(B, M), p.adjoint(f.reshape(-1))
    for i in range(B):
        q = NFFT(N, n=n, m=3, precision="f64", device=dev).set_nodes(x[i * M:(i + 1) * M])
        for got, ref in ((fwd[i], q.forward(fh[i])), (adj[i], q.adjoint(f[i]))):
            if AMPS[i] == 0.0:
                assert not got.abs().any()
            else:
                s = 1.0 / AMPS[i]  # so that the norms' squares stay in range
                assert torch.linalg.norm((got - ref) * s) < TOL * torch.linalg.norm(ref * s), (N, AMPS[i])
        q.close()
    p.close()
