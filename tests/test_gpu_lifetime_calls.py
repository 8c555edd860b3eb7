"""Tensors that a plan on its private stream still uses are not given to another plan's next
output, whichever call used them and however many calls were issued since; a plan on a caller's
stream holds nothing, and nothing stays held once later calls find the work done."""
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def _plans(n=2):
    from cunfft_gb300.nfft import NFFT
    dev = torch.device("cuda:0")
    g = torch.Generator(device=dev).manual_seed(1)
    N, M = [48, 48, 48], 200000
    x = torch.rand(M, 3, generator=g, device=dev, dtype=torch.float64) - 0.5
    fh = torch.randn(N, generator=g, device=dev, dtype=torch.complex128)
    f = torch.randn(M, generator=g, device=dev, dtype=torch.complex128)
    ps = [NFFT(N, m=12, precision="f64", device=dev).set_nodes(x) for _ in range(n)]
    for p in ps:  # modules loaded, buffers made
        p.forward(fh), p.adjoint(f), p.node_gradient(fh, f), p.interp(p.spread(f))
        p.synchronize()
    return ps, x, fh, f


def _used(name, p, x, fh, f):
    """Addresses that the calls used and that nothing but the plan refers to any more."""
    if name == "two forwards":
        return {p.forward(fh).data_ptr(), p.forward(fh).data_ptr()}
    if name == "two adjoints":
        return {p.adjoint(f).data_ptr(), p.adjoint(f).data_ptr()}
    if name == "interp":
        g = torch.ones(p.n, dtype=torch.complex128, device=fh.device)
        return {p.interp(g).data_ptr()}
    if name == "node gradient":
        return {p.node_gradient(fh, f).data_ptr()}
    if name == "converted input":  # complex64 samples and coefficients are converted by the call
        small = f.to(torch.complex64)
        c = p._samples(small)
        at = c.data_ptr()
        del c  # the call's own conversion takes the block just released
        p.adjoint(small)
        p.adjoint(small)
        return {at}
    if name == "ndft":
        return {p.ndft_forward(fh).data_ptr()}
    a = x.clone()
    p.set_nodes(a)
    p.ndft_adjoint(f)
    p.set_nodes(x)  # the direct sums still read a
    return {a.data_ptr()}


@pytest.mark.parametrize("name", ["two forwards", "two adjoints", "interp", "node gradient", "converted input", "ndft", "old nodes"])
def test_no_block_in_use_is_another_plans_output(name):
    (a, b), x, fh, f = _plans()
    busy = [a.forward(fh) for _ in range(4)]  # a's stream stays behind the host
    used = _used(name, a, x, fh, f)
    kept = [b.forward(fh), b.adjoint(f), b.ndft_forward(fh) if name == "ndft" else b.forward(fh), b.node_gradient(fh, f),
            b.set_nodes(x).forward(fh)] + [torch.empty(200000 * 3, dtype=torch.float64, device="cuda:0") for _ in range(2)]
    assert not used & {t.data_ptr() for t in kept}
    del busy
    a.close()
    b.close()


def test_held_tensors_are_released():
    """Calls on a plan whose work is done do not pile up memory, and none stays with synchronize()."""
    import gc
    (p, other), x, fh, f = _plans()
    torch.cuda.synchronize()
    gc.collect()  # other tests' tensors
    before = torch.cuda.memory_allocated()
    one = p.forward(fh).nbytes + p.node_gradient(fh, f).nbytes + p.interp(torch.ones(p.n, dtype=torch.complex128, device="cuda:0")).nbytes
    for _ in range(60):
        p.forward(fh), p.node_gradient(fh, f), p.interp(torch.ones(p.n, dtype=torch.complex128, device="cuda:0"))
        torch.cuda.synchronize()
    assert torch.cuda.memory_allocated() - before < 3 * p._HELD_BYTES < 60 * (one + 16 * 96 ** 3)
    p.synchronize()
    assert torch.cuda.memory_allocated() == before and not p._live
    p.close()
    other.close()


def test_a_plan_alone_holds_nothing():
    import gc
    from cunfft_gb300.nfft import NFFT
    gc.collect()
    if sum(NFFT._private_plans.values()):
        pytest.skip("plans of other tests are still open")
    (p,), x, fh, f = _plans(1)
    for _ in range(3):
        p.forward(fh), p.adjoint(f), p.ndft_forward(fh[:1].expand_as(fh))
    assert not p._live and not p._open and not p._pending
    p.close()


def test_a_plan_on_a_callers_stream_holds_nothing():
    from cunfft_gb300.nfft import NFFT
    dev = torch.device("cuda:0")
    s = torch.cuda.Stream(dev)
    with torch.cuda.stream(s):
        p = NFFT([16, 16], precision="f64", device=dev, stream=s).set_nodes(torch.zeros(4, 2, dtype=torch.float64, device=dev))
        y = p.forward(torch.ones(16, 16, dtype=torch.complex128, device=dev))
        p.node_gradient(torch.ones(16, 16, dtype=torch.complex128, device=dev), y)
        assert not p._live and not p._open and not p._pending
    p.close()
