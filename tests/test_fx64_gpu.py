"""GPU tests of the FP64 line kernels in block fixed point (line_fx64.cuh):
precision against extended-precision FFTs (scipy on long double), lines of
very different scale side by side, and the values the fixed-point form leaves
to the FP64 body (non-finite, near overflow, near underflow).

Tolerance: the final rounding to double (0.3e-16 rms), the FP64 twiddles (up
to 1.1e-16 each, up to four stages and one four-step factor, 2.5e-16 in all)
and the fixed-point units (2^-57 of the line's largest value, 5 times its rms,
one per stage: 0.4e-16 each) give 3e-16; the bound is twice that, and below
what FP64 butterflies leave (5e-16 at 4096 points).
"""
import numpy as np
import pytest

import fft_gb300 as G

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
sfft = pytest.importorskip("scipy.fft")

TOL = 6e-16


@pytest.fixture(scope="module")
def dev():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    return torch.device("cuda:0")


def run(kind, dims, batch, arrays, dev):
    n = int(np.prod(dims))
    m = (G.half_elems(dims) if kind == "r" else n) * batch
    src = [torch.from_numpy(np.ascontiguousarray(a, np.float64).ravel()).to(dev) for a in arrays]
    out = [torch.empty(m, dtype=torch.float64, device=dev) for _ in range(1 if kind == "ri" else 2)]
    p = G.BatchPlan(kind, dims, batch, form="f64")
    p(*src, *out)
    got = [o.cpu().numpy().reshape(batch, -1) for o in out]
    return got[0] if kind == "ri" else got[0].astype(np.clongdouble) + 1j * got[1].astype(np.longdouble)


def rel(got, ref):
    """Worst relative L2 error over the transforms of a batch."""
    d = np.abs(got - ref)
    return float(np.max(np.sqrt((d * d).sum(1) / (np.abs(ref) ** 2).sum(1))))


# one line length per schedule (first radix 2, 4, 8; one to five stages), lines
# of one thread, part of a warp, one warp, several warps, and an odd batch
@pytest.mark.parametrize("logn", [3, 4, 5, 6, 7, 8, 9, 10, 11, 12, 13])
@pytest.mark.parametrize("kind", ["c", "ci"])
def test_lines(logn, kind, dev):
    n, batch = 1 << logn, 3
    rng = np.random.default_rng(logn)
    a, b = rng.standard_normal((2, batch, n))
    z = a.astype(np.clongdouble) + 1j * b.astype(np.longdouble)
    ref = sfft.fft(z) if kind == "c" else sfft.ifft(z) * n
    assert rel(run(kind, [n], batch, (a, b), dev), ref) <= TOL


@pytest.mark.parametrize("logn", [4, 6, 9, 12, 14])
def test_real_lines(logn, dev):
    n, batch = 1 << logn, 3
    rng = np.random.default_rng(logn)
    a = rng.standard_normal((batch, n))
    ref = sfft.rfft(a.astype(np.longdouble))
    got = run("r", [n], batch, (a,), dev)
    assert rel(got, ref) <= TOL
    sr, si = ref.real.astype(np.float64), ref.imag.astype(np.float64)
    si[:, 0] = np.nan     # the inverse reads only the real parts of the first and last bin
    si[:, -1] = np.inf
    back = run("ri", [n], batch, (sr, si), dev)
    z = sr.astype(np.clongdouble)
    z.imag[:, 1:-1] = si[:, 1:-1]
    assert rel(back, sfft.irfft(z, n) * n) <= TOL


# strided passes of each tile width, the transposing store and the four-step twiddle
@pytest.mark.parametrize("dims", [[8, 32], [16, 16], [256, 8], [512, 16], [1024, 8], [2048, 4], [1 << 14], [1 << 17]])
def test_strided(dims, dev):
    rng = np.random.default_rng(7)
    a, b = rng.standard_normal((2, 1, int(np.prod(dims))))
    z = (a.astype(np.clongdouble) + 1j * b.astype(np.longdouble)).reshape(dims)
    assert rel(run("c", dims, 1, (a, b), dev), sfft.fftn(z).reshape(1, -1)) <= TOL


# lines of 8192 points, the longest of one pass; axes of 2^20 points in three
@pytest.mark.parametrize("kind,dims,batch", [("c", [8192], 9), ("ci", [2, 8192], 5), ("c", [1 << 20], 8)])
def test_split_lines(kind, dims, batch, dev):
    rng = np.random.default_rng(5)
    a, b = rng.standard_normal((2, batch, int(np.prod(dims))))
    z = (a.astype(np.clongdouble) + 1j * b.astype(np.longdouble)).reshape([batch] + dims)[-2:]
    axes = tuple(range(1, len(dims) + 1))
    ref = sfft.fftn(z, axes=axes) if kind == "c" else sfft.ifftn(z, axes=axes, norm="forward")
    assert rel(run(kind, dims, batch, (a, b), dev)[-2:], ref.reshape(2, -1)) <= TOL


# spiky and smooth lines, and neighbours of other scales, up to the ends of the range
@pytest.mark.parametrize("n", [8, 64, 256, 4096])
def test_scales(n, dev):
    rng = np.random.default_rng(n)
    j = np.arange(n)
    rows = [np.eye(1, n, 3)[0] * 1e6 + rng.standard_normal(n), np.exp(-((j - n / 2) / (n / 16)) ** 2),
            np.cos(2 * np.pi * 3 * j / n), np.ones(n), np.zeros(n)]
    rows += [rng.standard_normal(n) * s for s in (1e-300, 1e-240, 1e-30, 1.0, 1e30, 1e280, 1e300)]
    a = np.stack(rows)
    b = np.roll(a, 1, axis=1)
    z = a.astype(np.clongdouble) + 1j * b.astype(np.longdouble)
    ref = sfft.fft(z)
    got = run("c", [n], len(rows), (a, b), dev)
    assert np.all(got[4] == 0)
    keep = np.arange(len(rows)) != 4
    # scaled by exact powers of two, so that the squares of the norm stay in range
    s = np.exp2(-np.floor(np.log2(np.abs(a[keep]).max(1))))[:, None]
    assert rel(got[keep] * s, ref[keep] * s) <= TOL


@pytest.mark.parametrize("n", [8, 32, 512, 4096])
def test_non_finite_lines_stay_their_own(n, dev):
    batch = 40
    rng = np.random.default_rng(n)
    a, b = rng.standard_normal((2, batch, n))
    a[5, 3], b[11, n - 1], a[17, 0] = np.inf, np.nan, -np.inf
    a[23] = 5e-320      # subnormal data
    b[23] = 0
    got = run("c", [n], batch, (a, b), dev)
    bad = [5, 11, 17]
    assert not np.isfinite(got[bad].real.astype(np.float64)).any(1).all() or np.isnan(got[bad]).any()
    assert not np.isfinite(got[bad].astype(np.complex128)).all(1).any()
    good = [i for i in range(batch) if i not in bad + [23]]
    z = a.astype(np.clongdouble) + 1j * b.astype(np.longdouble)
    assert rel(got[good], sfft.fft(z[good])) <= TOL
    assert abs(float(got[23, 0].real) - n * 5e-320) <= 5e-324 * n


# the standalone real pass (lines longer than one CTA): scales to the ends of
# the range side by side, and a line that is not finite
def test_long_real_lines(dev):
    n = 1 << 15
    rng = np.random.default_rng(1)
    scale = np.array([1.0, 1e-300, 1e300, 1e-3, 0.0, 1e5])
    a = rng.standard_normal((len(scale), n)) * scale[:, None]
    a[3, 100] = np.nan
    good = [0, 1, 2, 5]
    s = np.exp2(-np.floor(np.log2(np.abs(a[good]).max(1))))[:, None]
    ref = sfft.rfft(a[good].astype(np.longdouble))
    got = run("r", [n], len(scale), (a,), dev)
    assert rel(got[good] * s, ref * s) <= TOL
    assert np.all(got[4] == 0) and not np.isfinite(got[3].astype(np.complex128)).any()
    sr, si = ref.real.astype(np.float64), ref.imag.astype(np.float64)
    si[:, [0, -1]] = np.nan
    back = run("ri", [n], 4, (sr * 2.0 ** -20, si * 2.0 ** -20), dev)
    z = sr.astype(np.clongdouble)
    z.imag[:, 1:-1] = si[:, 1:-1]
    want = sfft.irfft(z * s, n) * n
    assert rel(back * s * 2.0 ** 20, want) <= TOL
