"""GPU tests of FP64 transforms of data that one value dominates or that has a
mean, against extended-precision FFTs (scipy on long double).

Tolerances.  Real inverses of the spectrum of data with a mean: bin 0 is the
largest value and about the outputs' rms, so each of the line's L values,
converted and passed through the pre-pass to 0.65 units (2^-59 of bin 0) per
component, counts in full: 0.65 sqrt(2 L) 2^-59 = 1.4e-16 at the longest line
of 8192 points; the later stages, whose product rounds at 2^-57 of the line's
largest, but on 1/8 of the values each, add 0.8e-16; the last rounding and the
twiddles 0.8e-16: 1.8e-16 in all.  The bound is 3e-16, what FP64 butterflies
leave at worst (2.6e-16), rounded up.
Bin 0 of a positive line with one large value, relative to itself: rounding
without a mean leaves 0.35 sqrt(L / 2) units of 2^-57, 1.6e-16 at 8192 points
(a mean of a quarter unit would leave 70e-16); the last rounding and a real
post-pass 1.5e-16 at most: the bound is 4e-16.
"""
import numpy as np
import pytest

import fft_gb300 as G
from test_fx64_gpu import rel, run

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
sfft = pytest.importorskip("scipy.fft")

TOL_MEAN = 3e-16
TOL_BIN0 = 4e-16


@pytest.fixture(scope="module")
def dev():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    return torch.device("cuda:0")


def spectra(name, batch, n, rng):
    if name == "power law":
        shape = (batch, n // 2 + 1)
        return (rng.standard_normal(shape) + 1j * rng.standard_normal(shape)) * (np.arange(n // 2 + 1) + 1.0) ** -1.5
    x = {"offset": 10 + rng.standard_normal((batch, n)), "image row": 128 + 40 * rng.standard_normal((batch, n)),
         "positive": rng.uniform(0, 1, (batch, n))}[name]
    return sfft.rfft(x.astype(np.longdouble)).astype(np.complex128)


# lines whose first stage is of radix 8 (2^9 and 2^12 points), 2 and 4; rows of
# part of a warp, a warp and several
@pytest.mark.parametrize("n", [16, 128, 512, 1024, 2048, 4096, 8192, 16384])
@pytest.mark.parametrize("name", ["offset", "image row", "positive", "power law"])
def test_real_inverse(name, n, dev):
    batch = 5
    X = spectra(name, batch, n, np.random.default_rng(n))
    z = X.astype(np.clongdouble)
    z.imag[:, [0, -1]] = 0
    assert rel(run("ri", [n], batch, (X.real, X.imag), dev), sfft.irfft(z, n) * n) <= TOL_MEAN


# the strided pass, and the standalone one of lines longer than a CTA's (one
# pass or more besides: as much again)
@pytest.mark.parametrize("dims", [[16, 8], [512, 16], [2048, 8], [4096, 8], [1 << 15], [1 << 17]])
def test_real_inverse_in_passes(dims, dev):
    rng = np.random.default_rng(3)
    x = 10 + rng.standard_normal(dims)
    axes = tuple(range(1, len(dims))) + (0,)   # the half spectrum is along axis 0
    X = sfft.rfftn(x.astype(np.longdouble), axes=axes).astype(np.complex128)
    got = run("ri", dims, 1, (X.real, X.imag), dev)
    ref = sfft.irfftn(X.astype(np.clongdouble), s=[dims[a] for a in axes], axes=axes, norm="forward")
    assert rel(got, ref.reshape(1, -1)) <= 2 * TOL_MEAN


@pytest.mark.parametrize("n", [64, 512, 1024, 4096, 8192])
@pytest.mark.parametrize("kind", ["c", "r"])
@pytest.mark.parametrize("spike", [300.0, 1e5])
def test_spike_on_positive_line(spike, kind, n, dev):
    batch = 5
    m = n if kind == "c" else 2 * n
    a = np.random.default_rng(n).uniform(0, 1, (batch, m))
    a[:, m // 3] = spike
    b = np.roll(a, 5, axis=1)
    ref = sfft.rfft(a.astype(np.longdouble)) if kind == "r" else sfft.fft(a.astype(np.longdouble) + 1j * b)
    got = run(kind, [m], batch, (a,) if kind == "r" else (a, b), dev)
    assert float(np.max(np.abs(got[:, 0] - ref[:, 0]) / np.abs(ref[:, 0]))) <= TOL_BIN0
    assert rel(got, ref) <= TOL_MEAN
