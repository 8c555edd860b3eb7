"""FP32 gridding of wide 3D windows on the shared-tile kernels: 18 to 24 taps (a plane's window
spread over all lanes) and 26 to 32 (the padded tile in slabs of planes), against the oracle.

Tolerance (relative l2): three taps of about 2^-22 each, sums of some 70 terms of random signs
(2^-22) and, spreading, up to a thousand nodes on a cell, 2^-20 at random signs."""
import numpy as np
import pytest

import oracle as O

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

TOL = 4e-6


@pytest.mark.parametrize("window", ["gaussian", "es"])
@pytest.mark.parametrize("N,n,m", [([18, 20, 22], [37, 41, 45], 8), ([20, 18, 20], None, 10), ([24, 22, 20], [48, 47, 41], 11),
                                   ([20, 18, 20], None, 12), ([17, 20, 30], [34, 41, 63], 13), ([20, 18, 17], None, 14),
                                   ([33, 18, 20], [66, 36, 40], 15), ([16, 16, 16], None, 15)])
def test_wide_windows(N, n, m, window):
    from cunfft_gb300.nfft import NFFT
    dev = torch.device("cuda:0")
    rng = np.random.default_rng(m + N[0])
    x = np.concatenate([rng.uniform(0.0, 0.02, (1037, 3)), rng.uniform(-0.5, 0.5, (900, 3))])
    x[:3], x[3:5], x[5] = -0.5, np.nextafter(0.5, 0), -0.0
    p = NFFT(N, n=n, m=m, precision="f32", device=dev, window=window).set_nodes(torch.from_numpy(x).to(dev))
    assert (p.spread_kernel(), p.interp_kernel()) == ("shared", "shared")
    g = rng.uniform(-1, 1, p.n) + 1j * rng.uniform(-1, 1, p.n)
    f = rng.uniform(-1, 1, len(x)) + 1j * rng.uniform(-1, 1, len(x))
    got = p.interp(torch.from_numpy(g).to(dev)).cpu().numpy()
    assert O.rel_l2(O.interp(x, g, N, p.n, m, window=window), got) < TOL
    got = p.spread(torch.from_numpy(f).to(dev)).cpu().numpy()
    assert O.rel_l2(O.spread(x, f, N, p.n, m, window=window), got) < TOL
    p.close()


def test_wide_window_node_gradient_and_batches():
    """Plans in slabs: uneven instances, and the node gradient, which has no slabs of its own."""
    from cunfft_gb300.nfft import NFFT
    dev = torch.device("cuda:0")
    rng = np.random.default_rng(3)
    N, m, Ms = [16, 18, 17], 12, [700, 0, 1, 300]
    x = torch.from_numpy(rng.uniform(-0.5, 0.5, (sum(Ms), 3))).to(dev)
    fh = torch.from_numpy(rng.uniform(-1, 1, [4] + N) + 1j * rng.uniform(-1, 1, [4] + N)).to(dev)
    f = torch.from_numpy(rng.uniform(-1, 1, sum(Ms)) + 1j * rng.uniform(-1, 1, sum(Ms))).to(dev)
    got = {}
    for prec in ("f32", "f64"):
        p = NFFT(N, m=m, precision=prec, batch=4, device=dev).set_nodes(x, Ms)
        got[prec] = [v.cpu().numpy() for v in (p.forward(fh), p.adjoint(f), p.node_gradient(fh, f))]
        p.close()
    for a, b in zip(got["f64"], got["f32"]):
        assert O.rel_l2(a, b) < TOL


def test_wide_window_infinite_value_stays_where_it_is():
    """An infinite grid value reaches the nodes whose windows hold it, as an infinity (its
    weight is positive), and no other."""
    from cunfft_gb300.nfft import NFFT
    dev = torch.device("cuda:0")
    for m in (8, 12):
        W, n = 2 * m + 2, 48
        x = torch.tensor([[0.2, 0.2, 0.2], [-0.2, -0.2, -0.2]], dtype=torch.float64, device=dev)
        p = NFFT([24] * 3, n=[n] * 3, m=m, precision="f32", device=dev).set_nodes(x)
        start = [int(np.rint(n * 0.2)) - m + n] * 3
        for last in (0, W - 1):  # the window's first and last cell
            g = torch.zeros(n, n, n, dtype=torch.complex64, device=dev)
            i = [(s + last) % n for s in start]
            g.real[i[0], i[1], i[2]] = float("inf")
            v = p.interp(g).cpu().numpy()
            other = (i[0] - (int(np.rint(-n * 0.2)) - 1 - m)) % n < W  # in the second node's window too (m = 12)
            assert np.isposinf(v[0].real) and (np.isposinf(v[1].real) if other else v[1] == 0), (m, last, v)
        p.close()
