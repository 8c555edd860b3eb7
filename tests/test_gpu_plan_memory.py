"""FP64 plans on power-of-two grids hold their grid, and in 1D above 4096 points the FFT's second
buffer, but no library FFT plan with a workspace that they never use.

Bound: grid (and second buffer), the roll-off table of 8 bytes per bandwidth, and an eighth of a
grid for small arrays and 2 MB pages."""
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N,grids", [([128, 128, 128], 1), ([1024, 1024], 1), ([1 << 22], 2)])
def test_plan_memory(N, grids):
    from cunfft_gb300.nfft import NFFT
    dev = torch.device("cuda:0")
    small = NFFT([16] * len(N), precision="f64", device=dev)  # modules and context memory
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info(dev)[0]
    p = NFFT(N, precision="f64", device=dev)
    used = before - torch.cuda.mem_get_info(dev)[0]
    one = 16
    for v in p.n:
        one *= v
    assert used < (grids + 0.125) * one + 8 * sum(N), (used, one)
    p.close()
    small.close()
