"""GPU parity of the cols passes of 512 and 1024 points with 32 points per
thread (line_wide.cuh) against 64-bit FFTs: whole and partial tiles, arrays the
TMA forms take and ones off a 16-byte boundary, split data and pairs, tile
counts below, inside and above the pipelined form's range.  Bound: the
relative L2 error all FP32 kernels are held to."""
import numpy as np
import pytest

import fft_gb300 as G

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")
TOL = 2e-6


def check(kind, dims, batch, fmt, off):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    n, h = int(np.prod(dims)), G.half_elems(dims)
    g = torch.Generator(device="cuda")
    g.manual_seed(n + batch)
    shift = lambda m: torch.empty(m + off, device="cuda")[off:]  # noqa: E731

    def arrays(z):   # complex or real values as the arrays of the format
        parts = [torch.view_as_real(z).reshape(-1)] if z.is_complex() and fmt else \
            [z.real.reshape(-1), z.imag.reshape(-1)] if z.is_complex() else [z.reshape(-1)]
        out = [shift(p.numel()) for p in parts]
        for o, p in zip(out, parts):
            o.copy_(p)
        return out + [None] * (2 - len(out))

    axes = tuple(range(1, len(dims) + 1))
    m = h if kind == "ri" else n
    re = torch.randn(batch, m, generator=g, device="cuda")
    z = re if kind == "r" else torch.complex(re, torch.randn(batch, m, generator=g, device="cuda"))
    half = [dims[0] // 2 + 1] + dims[1:]
    x = z.to(torch.float64 if kind == "r" else torch.complex128).reshape([batch] + (half if kind == "ri" else dims))
    if kind == "c":
        want = torch.fft.fftn(x, dim=axes)
    elif kind == "ci":
        want = torch.fft.ifftn(x, dim=axes, norm="forward")
    elif kind == "r":
        want = torch.fft.fftn(torch.fft.rfft(x, dim=1), dim=axes[1:]) if len(dims) > 1 else torch.fft.rfft(x, dim=1)
    else:
        x = torch.fft.ifftn(x, dim=axes[1:], norm="forward") if len(dims) > 1 else x
        x = x.clone()
        x[:, 0].imag = 0
        x[:, -1].imag = 0
        want = torch.fft.irfft(x, n=dims[0], dim=1, norm="forward")
    src = arrays(z)
    o = batch * (h if kind == "r" else n)
    dst = [shift(o), None] if kind == "ri" else [shift(2 * o), None] if fmt else [shift(o), shift(o)]
    G.BatchPlan(kind, dims, batch, fmt=fmt).launch(*src, *dst, stream=torch.cuda.current_stream())
    got = dst[0] if kind == "ri" else torch.view_as_complex(dst[0].clone().reshape(-1, 2)) if fmt else torch.complex(*dst)
    err = float((got.to(want.dtype) - want.reshape(-1)).norm() / want.norm())
    assert err <= TOL, err


@pytest.mark.parametrize("off", [0, 1])
@pytest.mark.parametrize("fmt", [0, 1])
@pytest.mark.parametrize("kind,dims,batch", [
    ("c", [512, 2], 3), ("ci", [512, 4], 5), ("c", [512, 8], 3), ("ci", [512, 16], 1), ("c", [512, 64], 7),
    ("c", [1024, 2], 3), ("ci", [1024, 4], 3), ("c", [1024, 8], 1), ("c", [1024, 32], 5), ("ci", [2, 1024, 16], 3),
    ("c", [1 << 18], 3), ("ci", [1 << 19], 2), ("c", [1 << 20], 1),
    ("r", [1024, 2], 3), ("r", [1024, 32], 3), ("ri", [1024, 4], 3), ("ri", [1024, 16], 5),
    ("r", [2048, 2], 3), ("r", [2048, 16], 3), ("ri", [2048, 4], 3), ("ri", [2048, 16], 3),
    ("r", [4096, 4], 3), ("r", [4096, 32], 1), ("r", [1 << 20], 2), ("ri", [1 << 19], 2), ("ri", [1 << 20], 2),
    ("ri", [1 << 21], 1)])
def test_wide(kind, dims, batch, fmt, off):
    check(kind, dims, batch, fmt, off)


# rows: whole and partial CTAs (8 and 4 lines each)
@pytest.mark.parametrize("off", [0, 1])
@pytest.mark.parametrize("fmt", [0, 1])
@pytest.mark.parametrize("kind,dims,batch", [
    ("c", [512], 1), ("ci", [512], 7), ("c", [512], 8), ("c", [512], 1001), ("c", [1024], 1), ("ci", [1024], 3),
    ("c", [1024], 4), ("ci", [1024], 1001), ("r", [2048], 1), ("r", [2048], 3), ("r", [2048], 1001), ("r", [1024], 5),
    ("c", [4, 512], 3), ("ci", [8, 1024], 3),
    ("c", [8192], 1), ("ci", [8192], 5), ("c", [16384], 1), ("ci", [16384], 3), ("r", [16384], 1), ("r", [16384], 5),
    ("r", [32768], 3), ("ri", [16384], 3), ("ri", [32768], 3)])
def test_rows(kind, dims, batch, fmt, off):
    check(kind, dims, batch, fmt, off)


# 8-line tiles per launch on 304 CTA slots: one below and at two per slot, ten
# and one tile more
@pytest.mark.parametrize("kind,dims,batch", [
    ("c", [1024, 8], 607), ("c", [1024, 8], 608), ("ci", [1024, 8], 3040), ("c", [1024, 8], 3041),
    ("ri", [2048, 8], 607), ("ri", [2048, 8], 609), ("ci", [8, 1024, 64], 15)])
def test_tile_counts(kind, dims, batch):
    check(kind, dims, batch, 0, 0)
