"""Alternating node sets of different sizes allocate their bins once: items are shorter for fewer
nodes, so a smaller set can have more of them than a larger one.  The allocations of a child
process are counted by the host-side fault injection (CUNFFT_X_FAULT_ALLOC=k fails the k-th)."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

CHILD = r"""
import sys
sys.path.insert(0, ROOT)
import torch
from cunfft_gb300 import _native as nat
from cunfft_gb300.nfft import NFFT
g = torch.Generator(device="cuda:0").manual_seed(1)
sets = [torch.rand(M, DIM, generator=g, device="cuda:0", dtype=torch.float64) - 0.5 for M in (100000, 19000, 100000, 37000, 40000, 300, 99999)]
p = NFFT([40] * DIM, m=2, precision=PREC, device="cuda:0")
done = 0
try:
    for k in range(2):
        for x in sets:
            p.set_nodes(x)
            p.synchronize()
            done += 1
except nat.CunfftError as e:
    assert e.status == nat.ALLOC_FAILED
print("sets", done)
"""


def _sets(k, d, prec):
    code = CHILD.replace("ROOT", repr(ROOT)).replace("DIM", str(d)).replace("PREC", repr(prec))
    r = subprocess.run([sys.executable, "-c", code], env=dict(os.environ, CUNFFT_X_FAULT_ALLOC=str(k)), capture_output=True,
                       text=True, timeout=300)
    if "sets" not in r.stdout:  # the plan's own allocations come first
        return -1
    return int(r.stdout.split()[-1])


@pytest.mark.parametrize("d,prec,first", [(1, "f64", 17), (2, "f32", 22), (3, "f32", 16)])
def test_one_allocation_for_alternating_sets(d, prec, first):
    """`first`: about the last allocation of the plan's and the first set's."""
    got = [_sets(k, d, prec) for k in range(first, first + 4)]
    assert got[0] <= 0 and got[-1] == 14 and not any(0 < v < 14 for v in got), got
