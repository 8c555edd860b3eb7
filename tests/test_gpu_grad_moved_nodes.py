"""The node gradient is taken at the coordinates as they are at the call: nodes changed in place
since they were bound, against a plan bound to the new ones.  The FP32 form's tiles hold the
windows of the binning; nodes that left theirs take their own.

Tolerance: both forms round taps and sums to FP32 in the same way, 1e-5."""
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("window", ["gaussian", "es"])
@pytest.mark.parametrize("prec", ["f32", "f64"])
@pytest.mark.parametrize("N,n,batch", [([300], None, 1), ([40, 50], None, 1), ([33, 20], [67, 42], 3), ([16, 12, 20], None, 1), ([9, 14, 11], [19, 29, 23], 2)])
def test_nodes_changed_in_place(N, n, batch, prec, window):
    from cunfft_gb300.nfft import NFFT
    dev = torch.device("cuda:0")
    g = torch.Generator(device=dev).manual_seed(len(N))
    M, d = 900, len(N)
    x = torch.rand(batch * M, d, generator=g, device=dev, dtype=torch.float64) - 0.5
    cd = torch.complex64 if prec == "f32" else torch.complex128
    fh = torch.randn([batch] + N, generator=g, device=dev, dtype=cd)
    gf = torch.randn(batch * M, generator=g, device=dev, dtype=cd)
    p, q = (NFFT(N, n=n, m=4, precision=prec, batch=batch, device=dev, window=window) for _ in range(2))
    p.set_nodes(x, [M] * batch)
    step = torch.randn(batch * M, d, generator=g, device=dev, dtype=torch.float64) * 0.01
    step[:M // 2] = 0  # most of these stay, the others move by some cells
    x += step
    x -= torch.floor(x + 0.5)
    q.set_nodes(x.clone(), [M] * batch)
    ref = q.node_gradient(fh, gf)
    assert torch.linalg.norm(p.node_gradient(fh, gf) - ref) < 1e-5 * torch.linalg.norm(ref)
    p.close()
    q.close()


@pytest.mark.parametrize("m", [8, 11])
def test_wide_windows_are_not_slower_than_fp64(m):
    """3D windows above 16 taps: on staged tiles the FP32 gradient took up to six times the FP64
    form's time (37 against 6 ms at m = 11), thread per node half of it."""
    from cunfft_gb300.nfft import NFFT
    dev = torch.device("cuda:0")
    g = torch.Generator(device=dev).manual_seed(1)
    x = torch.rand(20000, 3, generator=g, device=dev, dtype=torch.float64) - 0.5
    took = {}
    for prec, cd in (("f32", torch.complex64), ("f64", torch.complex128)):
        p = NFFT([40] * 3, m=m, precision=prec, device=dev).set_nodes(x)
        fh, gf = torch.ones(40, 40, 40, dtype=cd, device=dev), torch.ones(20000, dtype=cd, device=dev)
        times = []
        for _ in range(6):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            torch.cuda.synchronize()
            a.record()
            p.node_gradient(fh, gf)
            b.record()
            torch.cuda.synchronize()
            times.append(a.elapsed_time(b))
        took[prec] = min(times)
        p.close()
    assert took["f32"] < took["f64"], took
