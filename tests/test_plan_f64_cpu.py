"""CPU emulation of the FP64 plans that split by batch: axes of 2^20 points and
more in three passes from 2^23 points in all; either side of the line, and the
scratch bound beyond which the plan keeps the form with less scratch.  Lines of
8192 points stay in one pass, without scratch."""
import numpy as np
import pytest

import fft_gb300 as G
from oracle import oracle as O
from plan_emulator import describe, run

F = G.FORM_F64


@pytest.mark.parametrize("kind,dims,batch,fmt,passes", [
    ("c", [8192], 9, 0, 1), ("ci", [2, 8192], 4, 0, 2), ("c", [2, 8192], 3, 1, 2), ("c", [1 << 20], 8, 0, 3)])
def test_emulation(kind, dims, batch, fmt, passes):
    desc = describe(kind, dims, batch, fmt | F)
    assert len(desc["ops"]) == passes
    n = int(np.prod(dims))
    rng = np.random.default_rng(n + batch)
    a, b = rng.standard_normal((2, n * batch))
    got = run(desc, a, b)
    z = (a + 1j * b).reshape([batch] + dims)
    axes = tuple(range(1, len(dims) + 1))
    ref = np.fft.fftn(z, axes=axes) if kind == "c" else np.fft.ifftn(z, axes=axes) * n
    assert O.rel_l2(got, (ref.real.ravel(), ref.imag.ravel())) < 1e-12


def test_scratch_bounds():
    count = lambda kind, dims, batch: len(describe(kind, dims, batch, F)["ops"])  # noqa: E731
    assert describe("c", [8192], 2048, F)["scratch_elems"] == 0
    assert count("c", [1 << 20], 7) == 2 and count("c", [1 << 20], 128) == 3 and count("c", [1 << 20], 129) == 2
    assert count("c", [1 << 22], 1) == 2 and count("c", [1 << 22], 2) == 3
    assert count("c", [1 << 19], 64) == 2
