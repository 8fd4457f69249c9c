"""The exchange layouts of the 512- and 1024-point cols kernels with 32 points
per thread (line_wide.cuh, and the pipelined 1024-point form in
line_fft_pipe.cuh), restated: injective, inside the buffer, and the two stages
compute the DFT through them.  A half-warp's 8-byte accesses (a warp's 4-byte
ones in the pipelined form) hit distinct banks."""
import numpy as np
import pytest

CASES = [(9, 8), (9, 16), (10, 8)]


def rows(logl, C):
    return (1 << logl) + (32 if C == 8 else 0)


def idx(logl, C, xor, c, j):
    r1 = (1 << logl) // 32
    row = j + j // r1 if C == 8 else j
    col = c if not xor else (c ^ ((j >> 1) & 7) if C == 8 else c ^ (j & 15))
    return row * C + col


def accesses(logl, C):
    """(element of thread t) per access of the cols mapping: the scatter's and the gather's."""
    L = 1 << logl
    T, r1 = L // 32, L // 32
    out = []
    for u in range(32 // r1):
        for r in range(r1):
            out.append(lambda t, u=u, r=r: (t + T * u) * r1 + r)
    for e in range(32):
        out.append(lambda t, e=e: t + T * e)
    return out


@pytest.mark.parametrize("logl,C", CASES)
@pytest.mark.parametrize("xor", [False, True])
def test_positions_and_banks(logl, C, xor):
    L, T = 1 << logl, (1 << logl) // 32
    c, j = np.meshgrid(np.arange(C), np.arange(L))
    pos = idx(logl, C, xor, c.ravel(), j.ravel())
    assert len(np.unique(pos)) == L * C and pos.min() >= 0 and pos.max() < rows(logl, C) * C
    tid = np.arange(T * C)
    for acc in accesses(logl, C):
        p = idx(logl, C, xor, tid % C, acc(tid // C))
        for half in p.reshape(-1, 16):
            assert len(np.unique(half % 16)) == 16
    if xor:   # the transposing store reads along lines: T threads per line
        for e in range(32):
            p = idx(logl, C, xor, tid // T, tid % T + T * e)
            for half in p.reshape(-1, 16):
                assert len(np.unique(half % 16)) == 16


@pytest.mark.parametrize("logl", [9, 10])
def test_rows(logl):
    L, T = 1 << logl, (1 << logl) // 32
    C = 128 // T
    pos = lambda c, j: c * (L + 32) + j + j // T  # noqa: E731  (T = R1)
    c, j = np.meshgrid(np.arange(C), np.arange(L))
    p = pos(c.ravel(), j.ravel())
    assert len(np.unique(p)) == L * C and p.max() < C * (L + 32)
    tid = np.arange(T * C)
    for acc in accesses(logl, C):
        for half in pos(tid // T, acc(tid % T)).reshape(-1, 16):
            assert len(np.unique(half % 16)) == 16


# 8192- and 16384-point rows: three stages (8 or 16, 32, 32 points)
@pytest.mark.parametrize("logl", [13, 14])
def test_long_rows(logl):
    L, T, r1 = 1 << logl, (1 << logl) // 32, (1 << logl) // 1024
    pos = lambda j: j + (j >> 4) + ((j >> 8) << 3)  # noqa: E731
    p = pos(np.arange(L))
    assert len(np.unique(p)) == L and p.max() < L + L // 16 + 8 * (L // 256)
    t = np.arange(T)
    acc = [(t + T * u) * r1 + r for u in range(32 // r1) for r in range(r1)]
    acc += [(t // r1) * (32 * r1) + t % r1 + r * r1 for r in range(32)] + [t + T * e for e in range(32)]
    for j in acc:
        for half in pos(j).reshape(-1, 16):
            assert len(np.unique(half % 16)) == 16
    rng = np.random.default_rng(logl)
    x = rng.standard_normal(L) + 1j * rng.standard_normal(L)
    b1, b2, out = (np.empty(L, complex) for _ in range(3))
    for t in range(T):
        v = x[t + T * np.arange(32)]
        for u in range(32 // r1):
            b = t + T * u
            b1[b * r1:(b + 1) * r1] = np.fft.fft(v[u + (32 // r1) * np.arange(r1)])
    r = np.arange(32)
    for t in range(T):
        k = t % r1
        b2[(t // r1) * 32 * r1 + k + r * r1] = np.fft.fft(b1[t + T * r] * np.exp(-2j * np.pi * r * k / (32 * r1)))
    for t in range(T):
        out[t + T * r] = np.fft.fft(b2[t + T * r] * np.exp(-2j * np.pi * r * t / L))
    assert np.abs(out - np.fft.fft(x)).max() < 1e-9


def test_pipelined_1024():
    T, C = 32, 8
    tid = np.arange(T * C)
    t, c = tid // C, tid % C
    row = lambda j: j + j // 32  # noqa: E731
    for e in range(32):
        for j, r in ((32 * t + e, 33 * t + e), (t + 32 * e, t + 33 * e)):   # scatter, gather: base + offset
            assert np.array_equal(row(j), r) and r.max() < 1024 + 32
            for warp in (r * C + c).reshape(-1, 32):
                assert len(np.unique(warp % 32)) == 32


@pytest.mark.parametrize("logl", [9, 10])
def test_two_stages_are_the_dft(logl):
    L = 1 << logl
    T, r1 = L // 32, L // 32
    rng = np.random.default_rng(logl)
    x = rng.standard_normal(L) + 1j * rng.standard_normal(L)
    buf = np.empty(L, complex)
    for t in range(T):
        v = x[t + T * np.arange(32)]
        for u in range(32 // r1):
            b = t + T * u
            buf[b * r1:(b + 1) * r1] = np.fft.fft(v[u + (32 // r1) * np.arange(r1)])
    out = np.empty(L, complex)
    for t in range(T):
        v = buf[t + T * np.arange(32)] * np.exp(-2j * np.pi * np.arange(32) * t / L)
        out[t + T * np.arange(32)] = np.fft.fft(v)
    assert np.abs(out - np.fft.fft(x)).max() < 1e-10
