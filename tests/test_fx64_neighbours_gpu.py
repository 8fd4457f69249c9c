"""GPU tests that an FP64 line's result is its own: bit for bit the same beside
lines that the fixed-point form leaves to the FP64 body (non-finite, near the
ends of the range, subnormal), beside ordinary ones, and where in its batch it
sits; and that a line goes by its largest value, however small a thread's are."""
import numpy as np
import pytest

import fft_gb300 as G
from test_fx64_gpu import TOL, rel, run

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
sfft = pytest.importorskip("scipy.fft")


@pytest.fixture(scope="module")
def dev():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    return torch.device("cuda:0")


def odd_data(m, rng):
    """Transforms of m values that go to the FP64 body."""
    rows = rng.standard_normal((5, m)) * np.array([1.0, 1.0, 1e-260, 1e305, 0.0])[:, None]
    rows[0, m // 3], rows[1, m - 1], rows[4, m // 2] = np.nan, np.inf, 5e-320
    return rows


# rows of one thread, part of a warp, a warp and several; strided tiles, whose
# lines belong to several transforms; the transposing store
@pytest.mark.parametrize("dims", [[8], [16], [64], [128], [256], [512], [1024], [4096], [4, 4], [16, 2], [64, 2],
                                  [256, 2], [512, 4], [1024, 2], [2048, 2], [1 << 14]])
@pytest.mark.parametrize("kind", ["c", "ci", "r", "ri"])
@pytest.mark.filterwarnings("ignore:invalid value")
def test_neighbours(kind, dims, dev):
    n = int(np.prod(dims))
    m = G.half_elems(dims) if kind == "ri" else n
    batch = max(5, min(64, 4096 // n))
    rng = np.random.default_rng(n)
    arrays = rng.standard_normal((1 if kind == "r" else 2, batch, m))
    want = run(kind, dims, batch, arrays, dev)
    assert np.isfinite(want.astype(np.complex128)).all()
    assert np.array_equal(run(kind, dims, batch, np.roll(arrays, 3, axis=1), dev), np.roll(want, 3, axis=0))
    odd = odd_data(m, rng)
    for start in range(5):   # every other transform one of them, a different one first each time
        mixed = arrays.copy()
        at = np.arange(start % 2, batch, 2)
        mixed[0, at] = odd[(at + start) % 5]
        got = run(kind, dims, batch, mixed, dev)
        rest = np.setdiff1d(np.arange(batch), at)
        assert np.array_equal(got[rest], want[rest])
        for i in at[:5]:     # and these as they are alone
            one = run(kind, dims, 1, mixed[:, i:i + 1], dev)
            assert np.array_equal(got[i].astype(np.complex128), one[0].astype(np.complex128), equal_nan=True)


# a decayed tail: values of whole threads below the range, the line's largest not
@pytest.mark.parametrize("n", [64, 512, 4096])
@pytest.mark.parametrize("kind", ["c", "r"])
def test_decayed_tail(kind, n, dev):
    batch = 3
    m = n if kind == "c" else 2 * n
    a = np.exp(-700.0 * np.arange(m) / m) * np.random.default_rng(n).uniform(0.5, 1, (batch, m))
    assert a[:, -m // 8:].max() < 2.0 ** -823
    b = np.roll(a, 1, axis=1)
    ref = sfft.rfft(a.astype(np.longdouble)) if kind == "r" else sfft.fft(a.astype(np.longdouble) + 1j * b)
    got = run(kind, [m], batch, (a,) if kind == "r" else (a, b), dev)
    assert rel(got, ref) <= TOL / 2   # (the FP64 body leaves 2.2e-16)
