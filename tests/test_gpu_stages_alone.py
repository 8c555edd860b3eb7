"""The FP64 form's gridding stages on their own keep FP64's relative precision of every single
value: cells at a window's edge, nodes and samples far smaller than their neighbours, clustered
nodes.  Values and samples are positive, so that nothing cancels.

Tolerance (relative, per value): the taps' recurrence leaves up to 4 W 2^-53 per tap and dimension
on both sides, 1e-13 for W = 32 in 3D, and sums of up to 2000 terms as much again.  ES taps near
the window's edge go with the square root of 1 - y^2 / alpha^2, whose rounding they magnify by up
to beta / (2 sqrt(z)) with z > 1e-5 for the taps drawn: 1e-11."""
import ctypes

import numpy as np
import pytest

import oracle as O

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

CASES = [([40], 2), ([300], 6), ([600], 15), ([33, 20], 3), ([60, 70], 6), ([40, 90], 7), ([40, 33], 15), ([12, 20, 18], 1), ([24, 20, 33], 6),
         ([20, 18, 20], 7), ([18, 20, 22], 8), ([16, 20, 24], 12), ([16, 17, 20], 15)]
TOL = {"gaussian": 5e-13, "es": 1e-11}


def _close(ref, got, tol):
    hit = ref != 0
    assert hit.any() and not got[~hit].any()
    for a, b in ((ref.real, got.real), (ref.imag, got.imag)):
        assert (np.abs(a - b)[hit] <= tol * a[hit]).all()


def _positive(shape, rng):
    return rng.uniform(0.5, 1.5, shape) + 1j * rng.uniform(0.5, 1.5, shape)


@pytest.mark.parametrize("window", ["gaussian", "es"])
@pytest.mark.parametrize("N,m", CASES)
def test_every_value_has_its_own_precision(N, m, window):
    from cunfft_gb300.nfft import NFFT
    dev = torch.device("cuda:0")
    rng = np.random.default_rng(10 * len(N) + m)
    d = len(N)
    # a few nodes of magnitude one and many small ones in the same tile, lone nodes elsewhere
    x = np.concatenate([rng.uniform(0.0, 0.02, (700, d)), rng.uniform(-0.5, 0.5, (9, d))])
    p = NFFT(N, m=m, precision="f64", device=dev, window=window).set_nodes(torch.from_numpy(x).to(dev))
    f = _positive(len(x), rng) * 10.0 ** rng.integers(-30, 1, len(x))
    f[0] = 1e5 * (1 + 1j)
    for s in (f, np.where(np.arange(len(x)) == 0, 0, f)):
        _close(O.spread(x, s, N, p.n, m, window=window), p.spread(torch.from_numpy(s).to(dev)).cpu().numpy(), TOL[window])
    one = np.zeros(len(x), dtype=complex)
    one[-1] = 1 + 2j  # one lone node: every cell of its window, edges and corners
    _close(O.spread(x, one, N, p.n, m, window=window), p.spread(torch.from_numpy(one).to(dev)).cpu().numpy(), TOL[window])
    g = _positive(p.n, rng) * 10.0 ** rng.integers(-30, 1, p.n)
    g[(np.indices(p.n).sum(0) % 7) != 0] *= 1e-20
    _close(O.interp(x, g, N, p.n, m, window=window), p.interp(torch.from_numpy(g).to(dev)).cpu().numpy(), TOL[window])
    p.close()


def test_spreading_without_allocation_as_well():
    from cunfft_gb300 import _native as nat
    dev = torch.device("cuda:0")
    rng = np.random.default_rng(4)
    N, n, M = [20, 24], [64, 64], 1500
    x = rng.uniform(-0.1, 0.1, (M, 2))
    f = _positive(M, rng) * 10.0 ** rng.integers(-30, 1, M)
    g = torch.zeros(n, dtype=torch.complex128, device=dev)
    xt, ft = torch.from_numpy(x).to(dev), torch.from_numpy(f).to(dev)
    fn = nat.lib().cunfft_x_spread_noalloc
    vp = lambda t: ctypes.c_void_p(t.data_ptr())
    stream = ctypes.c_void_p(torch.cuda.current_stream(dev).cuda_stream)
    assert fn(2, (ctypes.c_int64 * 2)(*N), None, 5, nat.F64, ctypes.c_int64(M), vp(xt), vp(ft), vp(g), stream, None) == nat.SUCCESS
    torch.cuda.synchronize()
    _close(O.spread(x, f, N, n, 5), g.cpu().numpy(), TOL["gaussian"])


@pytest.mark.parametrize("N,m", CASES)
def test_transforms_of_every_width(N, m):
    """The transforms' fixed-point kernels, against the oracle (relative l2, its taps' 1e-13 times
    the roll-off's amplification of (1 + m / 6) per dimension)."""
    from cunfft_gb300.nfft import NFFT
    dev = torch.device("cuda:0")
    rng = np.random.default_rng(7 * len(N) + m)
    x = np.concatenate([rng.uniform(0.0, 0.02, (700, len(N))), rng.uniform(-0.5, 0.5, (900, len(N)))])
    x[:3], x[3:5], x[5] = -0.5, np.nextafter(0.5, 0), -0.0
    fh = rng.uniform(-1, 1, N) + 1j * rng.uniform(-1, 1, N)
    f = rng.uniform(-1, 1, len(x)) + 1j * rng.uniform(-1, 1, len(x))
    tol = 1e-13 * (1 + m / 6) ** len(N)
    p = NFFT(N, m=m, precision="f64", device=dev).set_nodes(torch.from_numpy(x).to(dev))
    assert O.rel_l2(O.nfft_forward(x, fh, N, m=m), p.forward(torch.from_numpy(fh).to(dev)).cpu().numpy()) < tol
    assert O.rel_l2(O.nfft_adjoint(x, f, N, m=m), p.adjoint(torch.from_numpy(f).to(dev)).cpu().numpy()) < tol
    p.close()
