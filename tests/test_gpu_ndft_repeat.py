"""The direct NDFT repeats itself bit by bit, also where its sums are split over CTAs, under stream
capture gives the same sums, and keeps infinities and the full FP64 range.

Tolerances: captured and plain sums differ in the order of addition only, 1e-13."""
import numpy as np
import pytest

import oracle as O

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def _case(N, M, seed=0, stream=None, batch=1):
    from cunfft_gb300.nfft import NFFT
    dev = torch.device("cuda:0")
    rng = np.random.default_rng(seed)
    rand = lambda s: torch.from_numpy(rng.uniform(-1, 1, s) + 1j * rng.uniform(-1, 1, s)).to(dev)
    x = torch.from_numpy(rng.uniform(-0.5, 0.5, (M * batch, len(N)))).to(dev)
    p = NFFT(N, m=2, precision="f64", device=dev, stream=stream, batch=batch).set_nodes(x, [M] * batch)
    return p, x, rand(([batch] if batch > 1 else []) + N), rand(M * batch)


@pytest.mark.parametrize("N,M,batch", [([64, 64], 4096, 1), ([50], 300, 1), ([700], 90, 1), ([20, 33], 1000, 3), ([6, 10, 12], 700, 1)])
def test_same_bits_every_time(N, M, batch):
    p, x, fh, f = _case(N, M, batch=batch)
    a, b = p.ndft_forward(fh), p.ndft_adjoint(f)
    for _ in range(12):
        assert torch.equal(a, p.ndft_forward(fh)) and torch.equal(b, p.ndft_adjoint(f))
    p.close()


def test_under_capture():
    s = torch.cuda.Stream()
    with torch.cuda.stream(s):
        p, x, fh, f = _case([40, 30], 900, stream=s)
        a, b = p.ndft_forward(fh), p.ndft_adjoint(f)
        s.synchronize()
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=s):
            c, d = p.ndft_forward(fh), p.ndft_adjoint(f)
        g.replay()
        s.synchronize()
    assert torch.linalg.norm(c - a) < 1e-13 * torch.linalg.norm(a) and torch.linalg.norm(d - b) < 1e-13 * torch.linalg.norm(b)
    p.close()


@pytest.mark.parametrize("N,M", [([40], 200), ([64, 64], 4096), ([16], 130000), ([2000, 300], 20), ([5, 6, 7], 150)])
def test_infinities_stay_infinite(N, M):
    """An infinite real or imaginary part makes both parts of every result infinite, but for the
    frequency zero, whose phase has a sine of zero (times infinity: not a number)."""
    p, x, fh, f = _case(N, M, 1)
    fh.reshape(-1)[3] = complex(float("inf"), 0.0)
    assert torch.isinf(torch.view_as_real(p.ndft_forward(fh))).all()
    f[5] = complex(0.0, float("-inf"))
    v = torch.view_as_real(p.ndft_adjoint(f))
    zero = tuple(n // 2 for n in N)
    assert not torch.isfinite(v[zero]).all()
    v[zero] = float("inf")
    assert torch.isinf(v).all()
    p.close()


@pytest.mark.parametrize("N", [[40], [16, 30]])
def test_sums_near_the_largest_number(N):
    """Terms of 1.2e308 whose pair sums or differences overflow while the sum does not."""
    p, x, fh, f = _case(N, 300, 2)
    small = torch.zeros_like(fh)
    at = fh.numel() // 2
    small.reshape(-1)[at - 1], small.reshape(-1)[at] = 1.2, -1.2  # frequencies -1 and 0
    ref = p.ndft_forward(small)
    got = p.ndft_forward(small * 1e308)
    ok = torch.view_as_real(ref).abs().amax(-1) < 1.5
    assert ok.any() and torch.isfinite(torch.view_as_real(got[ok])).all()
    assert ((got[ok] * 1e-308 - ref[ok]).abs() < 1e-14).all()
    p.close()


@pytest.mark.parametrize("N", [[30, 1], [9, 7, 1], [40, 1, 1], [1, 1], [1, 33, 1]])
def test_trailing_dimensions_of_one_coefficient(N):
    """Frequency zero only; the nodes keep their coordinates there (phases of k x rounded: 1e-12)."""
    p, x, fh, f = _case(N, 250, 3)
    xh = x.cpu().numpy()
    assert O.rel_l2(O.ndft_forward(xh, fh.cpu().numpy(), N), p.ndft_forward(fh).cpu().numpy()) < 1e-12
    got = p.ndft_adjoint(f).cpu().numpy()
    assert O.rel_l2(O.ndft_adjoint(xh, f.cpu().numpy(), N).reshape(got.shape), got) < 1e-12
    f[3] = float("inf")
    assert torch.isinf(torch.view_as_real(p.ndft_adjoint(f)).reshape(-1)[::2]).any()
    p.close()


@pytest.mark.parametrize("N,like,M,adjoint,factor", [([64], [8, 8], 100000, False, 1.5), ([20000, 1], [20000], 300, True, 3.0),
                                                     ([300, 1, 1], [300], 5000, True, 3.0)])
def test_few_rows_take_no_longer(N, like, M, adjoint, factor):
    """As long as another shape of as many terms (an eighth of the work was used at N = 64, a
    thirtieth with a last dimension of one)."""
    took = []
    for shape in (N, like):
        p, x, fh, f = _case(shape, M)
        times = []
        for _ in range(6):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            torch.cuda.synchronize()
            a.record()
            p.ndft_adjoint(f) if adjoint else p.ndft_forward(fh)
            b.record()
            torch.cuda.synchronize()
            times.append(a.elapsed_time(b))
        took.append(min(times))
        p.close()
    assert took[0] < factor * took[1], took
