"""GPU tests of plans launched with programmatic stream serialization: passes
queued back to back, between other kernels and inside a captured graph give
bit for bit what the same passes give one at a time."""
import numpy as np
import pytest

import fft_gb300 as G

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

# one case per kernel family: rows, staged short rows, TMA and pipelined cols,
# LSU cols (unaligned arrays: neighbouring tiles share sectors), plane-fused,
# four-step, paired real passes, standalone real pass, interleaved, FP64
CASES = [("c", [4096], 64, 0, None, 0), ("c", [64], 999, 0, None, 1), ("c", [256, 64, 32], 3, 0, None, 0),
         ("c", [64, 16, 128], 5, 0, None, 1), ("ci", [1024, 256], 8, 0, None, 0), ("c", [512, 64], 37, 1, None, 0),
         ("c", [65536], 9, 0, None, 1), ("r", [1 << 18], 4, 0, None, 0), ("ri", [1 << 18], 4, 0, None, 0),
         ("ri", [1 << 20], 2, 0, None, 0), ("r", [64, 128], 16, 0, None, 1), ("ri", [2048, 64], 2, 0, None, 0),
         ("c", [128, 1024], 2, 0, "f64", 0), ("ri", [64, 32, 16], 3, 0, "f64", 0), ("r", [1 << 16], 3, 0, "f64", 0)]


@pytest.fixture(scope="module")
def dev():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    return torch.device("cuda:0")


@pytest.mark.parametrize("kind,dims,batch,fmt,form,off", CASES)
def test_back_to_back_and_captured(kind, dims, batch, fmt, form, off, dev):
    n, h = int(np.prod(dims)), G.half_elems(dims)
    dt = torch.float64 if form else torch.float32
    w = 2 if fmt else 1
    m_in = (h if kind == "ri" else n) * batch * (w if kind != "r" else 1)
    m_out = (h if kind == "r" else n) * batch * (w if kind != "ri" else 1)
    g = torch.Generator(device=dev)
    g.manual_seed(3)
    new = lambda m: torch.randn(m + off, generator=g, device=dev, dtype=dt)[off:]  # noqa: E731
    src, dst = [new(m_in), new(m_in)], [new(m_out), new(m_out)]
    plan = G.BatchPlan(kind, dims, batch, fmt=fmt, form=form)
    args = [src[0], None if kind == "r" or fmt else src[1], dst[0], None if kind == "ri" or fmt else dst[1]]
    start = [x.clone() for x in src]
    reps = 6

    def step(wait):
        # the input changes before each pass, and each result is read after it
        s = torch.cuda.current_stream()
        acc = torch.zeros_like(dst[0])
        for x, y in zip(src, start):
            x.copy_(y)
        for _ in range(reps):
            src[0].mul_(0.5)
            plan.launch(*args, stream=s)
            if wait:
                torch.cuda.synchronize()
            plan.launch(*args, stream=s)   # right behind its own twin, onto the same arrays
            if wait:
                torch.cuda.synchronize()
            acc += dst[0]
        return acc

    want = step(True)
    assert bool(torch.isfinite(want).all())
    assert torch.equal(step(False), want)
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        assert torch.equal(step(False), want)
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=side):
            got = step(False)
        for _ in range(2):
            graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(got, want)
