"""Outputs that are dropped while their plan's private stream may still write them are not given
to another plan's next call."""
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def test_dropped_outputs_do_not_become_another_plans():
    from cunfft_gb300.nfft import NFFT
    dev = torch.device("cuda:0")
    g = torch.Generator(device=dev).manual_seed(1)
    x = torch.rand(50000, 3, generator=g, device=dev, dtype=torch.float64) - 0.5
    fh = torch.randn(31, 54, 17, generator=g, device=dev, dtype=torch.complex64)
    f = torch.randn(50000, generator=g, device=dev, dtype=torch.complex64)
    a, b = (NFFT([31, 54, 17], n=[63, 109, 42], precision="f32", device=dev).set_nodes(x) for _ in range(2))
    for _ in range(3):
        used = {a.forward(fh).data_ptr(), a.adjoint(f).data_ptr()}
        kept = [b.forward(fh), b.adjoint(f)]
        assert not used & {t.data_ptr() for t in kept}
    a.close()
    b.close()


def test_the_kept_tensors_hold_no_autograd_graph():
    from cunfft_gb300.nfft import NFFT
    dev = torch.device("cuda:0")
    p = NFFT([16], precision="f64", device=dev).set_nodes(torch.zeros(4, 1, dtype=torch.float64, device=dev))
    v = (torch.ones(16, dtype=torch.complex128, device=dev, requires_grad=True) * 2)
    p.forward(v)
    assert all(t.grad_fn is None for pair in p._live.values() for t in pair)
    p.synchronize()
    assert not p._live
    p.close()
