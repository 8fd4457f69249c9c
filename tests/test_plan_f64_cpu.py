"""CPU emulation of the FP64 plans that split by batch: 8192-point lines in two
passes from 8 lines, axes of 2^20 points and more in three from 2^23 points in
all; either side of each line, and the scratch bounds beyond which the plan
keeps the form with less scratch."""
import numpy as np
import pytest

import fft_gb300 as G
from oracle import oracle as O
from plan_emulator import describe, run

F = G.FORM_F64


@pytest.mark.parametrize("kind,dims,batch,fmt,passes", [
    ("c", [8192], 7, 0, 1), ("c", [8192], 8, 0, 2), ("ci", [8192], 9, 1, 2), ("ci", [2, 8192], 4, 0, 3),
    ("c", [2, 8192], 3, 1, 2), ("c", [1 << 20], 8, 0, 3)])
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
    assert count("c", [8192], 1 << 15) == 2 and count("c", [8192], (1 << 15) + 1) == 1
    assert count("c", [1 << 20], 7) == 2 and count("c", [1 << 20], 128) == 3 and count("c", [1 << 20], 129) == 2
    assert count("c", [1 << 22], 1) == 2 and count("c", [1 << 22], 2) == 3
    assert count("c", [1 << 19], 64) == 2
