"""CPU tests of what the front end takes an address from: arrays whose memory
is the caller's, and nothing that only describes or copies some."""
import numpy as np
import pytest

import fft_gb300 as G


class Image:
    """An object whose array interface carries its data as bytes."""

    def __init__(self, **more):
        self.__array_interface__ = dict({"data": b"%pixels", "shape": (7,), "typestr": "|u1", "version": 3}, **more)


class Address:
    """One whose interface gives an address."""
    x = np.arange(4, dtype=np.float32)

    @property
    def __array_interface__(self):
        return self.x.__array_interface__


@pytest.mark.parametrize("a", [Image(), Image(data=(1234, False)), Address(), np.float32(1), np.float64(1.0),
                               b"bytes", bytearray(8), [1.0], 2.5], ids=lambda a: type(a).__name__)
def test_refused(a):
    with pytest.raises(TypeError):
        G.ptr(a)


def test_arrays(tmp_path):
    a = np.arange(24, dtype=np.float64).reshape(4, 6)
    np.save(tmp_path / "a.npy", a)

    class Sub(np.ndarray):
        pass

    for x in (a, a[1:], a[:, 2:], a.T, a[2, 3], np.float64(0) + a, a.view(Sub), np.ma.masked_array(a),
              np.load(tmp_path / "a.npy", mmap_mode="r"), np.array(1.0), np.empty(0)):
        if isinstance(x, np.ndarray):
            assert G.ptr(x) == x.ctypes.data
