"""GPU parity of complex axes above 2^22 points, whose first pass takes the
four-step twiddle as the hi/lo pair in each of its forms (TMA or LSU loads,
split planes or pairs, plan or queue).  The tolerance is that of the other
lengths: the pair's product adds one rounding (6e-8) to one of three passes."""
import numpy as np
import pytest

import fft_gb300 as G
from test_parity_gpu import check, inputs, run_plan

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


@pytest.fixture(scope="module")
def dev():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    return torch.device("cuda:0")


@pytest.mark.parametrize("kind,log,fmt,pad", [
    ("c", 23, 0, 0), ("ci", 23, 0, 1), ("c", 23, 1, 0), ("ci", 23, 1, 1), ("c", 24, 0, 0),
    ("ri", 24, 0, 0), ("ri", 24, 1, 1)])
def test_axes(kind, log, fmt, pad, dev):
    a, b = inputs(kind, [1 << log], log)
    check(kind, [1 << log], a, b, run_plan(kind, [1 << log], a, b, dev, fmt=fmt, pad=pad))


def test_queue(dev):
    n = 1 << 23
    a, b = inputs("c", [n], 3)
    s = [torch.from_numpy(x).to(dev) for x in (a, b)]
    d = [torch.empty(n, device=dev) for _ in range(4)]
    u = [torch.zeros(n + 1, device=dev)[1:] for _ in range(2)]
    for x, y in zip(u, s):
        x.copy_(y)
    q = G.Queue([("c", [n], *s, *d[:2]), ("c", [n], *u, *d[2:])])   # TMA loads; LSU loads
    q.run()
    torch.cuda.synchronize()
    for i in (0, 2):
        check("c", [n], a, b, tuple(x.cpu().numpy() for x in d[i:i + 2]))
