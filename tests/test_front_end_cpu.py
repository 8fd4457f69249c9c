"""CPU tests of the front end's array checks and addresses: what a plan object
checks per call is what the one-off check says for its shape."""
import numpy as np
import pytest

import fft_gb300 as G

torch = pytest.importorskip("torch")


@pytest.mark.parametrize("kind", ["c", "ci", "r", "ri"])
@pytest.mark.parametrize("dims,batch,fmt", [([1], 1, 0), ([8], 3, 0), ([4, 1, 8], 2, 0), ([16, 8], 5, 1)])
def test_wants(kind, dims, batch, fmt):
    n, h = int(np.prod(dims)), G.half_elems(dims)
    side = {"c": (n, n), "ci": (n, n), "r": (n, h), "ri": (h, n)}[kind]
    cplx = {"c": (1, 1), "ci": (1, 1), "r": (0, 1), "ri": (1, 0)}[kind]
    want = []
    for m, c in zip(side, cplx):
        want += [m * batch * (2 if c and fmt else 1), m * batch if c and not fmt else 0]
    assert G._wants(kind, dims, batch, fmt) == tuple(want)
    for new in (lambda m: np.zeros(m, np.float32), lambda m: torch.zeros(m)):
        arrays = [new(m) if m else None for m in want]
        G._check_arrays(tuple(want), "float32", arrays)
        for i, m in enumerate(want):
            if m:
                wrongs = [new(m)[:-1], arrays[i].astype(np.float64) if hasattr(arrays[i], "astype")
                          else arrays[i].double()]
                if m > 1:   # (a view of one element is contiguous at any stride)
                    wrongs.append(new(2 * m)[::2])
                for wrong in wrongs:
                    with pytest.raises(G.AfftError):
                        G._check_arrays(tuple(want), "float32", arrays[:i] + [wrong] + arrays[i + 1:])


def test_dtype_names():
    assert G._dtype_name(np.dtype("<f4")) == "float32" and G._dtype_name(torch.float64) == "float64"
    assert G._dtype_name(np.dtype(">f4")) not in ("float32", "float64")     # foreign byte order
    assert G._dtype_name(torch.float16) not in ("float32", "float64")
    assert np.dtype(">f4") not in G._FLOAT_DTYPES and torch.float16 not in G._FLOAT_DTYPES


def test_ptr():
    a = np.arange(8, dtype=np.float32)
    a.flags.writeable = False
    t = torch.zeros(8)
    assert G.ptr(a) == a.ctypes.data and G.ptr(a[2:]) == a.ctypes.data + 8
    assert G.ptr(t) == t.data_ptr() and G.ptr(t[3:]) == t.data_ptr() + 12
    assert G.ptr(None) is None and G.ptr(7) == 7
    with pytest.raises(TypeError):
        G.ptr("x")
