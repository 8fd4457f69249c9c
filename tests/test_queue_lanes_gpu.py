"""GPU test of queues launched behind one another: graphs of fewer, as many and
more kernel groups than lanes, run in rotation without waiting, leave bit for
bit what each leaves alone."""
import pytest

import fft_gb300 as G
from fft_gb300 import uneven as U

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("counts", [(1, 2, 3), (5, 13, 40), (120, 300, 7)])
def test_rotation(counts):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    dev = torch.device("cuda:0")
    queues = []
    for i, n in enumerate(counts):
        items = U.uneven_batch(n, seed=20 + i, max_log1d=17, side2d=(4, 10), side3d=(3, 6))
        buf, offs = U.allocate(items, dev, seed=i)
        q = G.Queue(U.descs(items, buf, offs))
        before = buf.clone()
        q.run()
        torch.cuda.synchronize()
        queues.append((q, buf, before, buf.clone()))
    for _, buf, before, _ in queues:
        buf.copy_(before)
    for _ in range(4):
        for q, _, _, _ in queues:
            q.run()
    torch.cuda.synchronize()
    for _, buf, _, want in queues:
        assert torch.equal(buf, want)
