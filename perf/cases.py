"""Transforms that are timed, each through the entry point a user's program calls.

A case is one of

- ``launch``: a ``BatchPlan`` whose arrays live on the GPU, enqueued on the
  program's stream (signal batches, images, volumes in a larger pipeline);
- ``call``: afft's own interface on device arrays, one transform per
  synchronous call;
- ``host``: the same interface on numpy arrays, as a program ported from afft
  calls it;
- ``queue``: many transforms of different sizes and kinds as one ``Queue``.

``kind`` is c, ci, r or ri (complex or real, ``i`` the inverse), or c+ci and
r+ri for a forward transform followed by the inverse of its result.  ``dims``
is the shape of one transform, ``batch`` how many lie back to back, ``bits``
32 or 64, ``inter`` whether complex arrays hold re,im pairs.
"""
import math
import random

import numpy as np
import torch

import fft_gb300 as G


def _case(name, api, kind, dims, batch=1, bits=32, inter=False):
    c = {"api": api, "kind": kind, "dims": dims, "batch": batch, "bits": bits, "inter": inter}
    return dict(c, name=name) if name else c


def listed():
    return [
        # one short transform and its inverse, call by call: launch and host latency
        _case("single_1024", "call", "c+ci", "1024"),
        # a ported afft program: one medium transform on host arrays
        _case("host_65536", "host", "c", "65536"),
        # spectrogram frames: many short real lines, an odd number of them
        _case("frames_r512", "launch", "r", "512", batch=30011),
        # channelised signal blocks: one pass over contiguous lines
        _case("lines_4096", "launch", "c", "4096", batch=16384),
        # long records as re,im pairs, transformed back: two passes per transform
        _case("records_65536_inter", "launch", "ci", "65536", batch=1001, inter=True),
        # long real records, there and back (convolution, filtering)
        _case("real_1m", "launch", "r+ri", "1048576", batch=64),
        # image filtering: a stack of camera frames as re,im pairs, odd count
        _case("images_512_inter", "launch", "c", "512x512", batch=37, inter=True),
        # one large real image and back, through afft's own calls
        _case("image_4096_real", "call", "r+ri", "4096x4096"),
        # one volume
        _case("volume_256", "launch", "c", "256x256x256"),
        # FP64 signal blocks
        _case("lines_4096_f64", "launch", "c", "4096", batch=4099, bits=64),
        # FP64 field solver: a real volume there and back
        _case("volume_real_f64", "launch", "r+ri", "128x128x256", batch=2, bits=64),
        # a server's mixed load: every kind, 1D 2^6..2^18, 2D 2^6..2^11, 3D 2^5..2^8 per side
        {"name": "queue_mixed", "api": "queue", "count": 3000, "mix": 5},
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def _shape(rng, log_total, sides):
    """`sides` powers of two whose product is 2^log_total, each side within the range the kinds support."""
    if sides == 1:
        return [log_total]
    while True:
        cut = [rng.randint(1, 11) for _ in range(sides)]
        if sum(cut) <= log_total + 1:
            return cut


def draw(rng):
    api = rng.choice(["launch"] * 7 + ["call"] * 2 + ["host", "queue"])
    if api == "queue":
        return {"api": "queue", "count": _log_int(rng, 40, 1500), "mix": rng.randrange(1 << 20)}
    kind = rng.choice(["c", "ci", "r", "ri", "c+ci", "r+ri"])
    bits = rng.choice([32, 32, 64])
    sides = rng.choice([1, 1, 2, 3])
    top = 20 if api == "host" else 22
    logs = _shape(rng, rng.randint(4, top), sides)
    points = 1 << sum(logs)
    batch = 1
    if api == "launch":
        most = (1 << 25) // points
        batch = _log_int(rng, 1, most) if most > 1 else 1
    return _case(None, api, kind, "x".join(str(1 << k) for k in logs), batch=batch, bits=bits, inter=rng.random() < 0.25)


# ---------------------------------------------------------------------------
# shapes
# ---------------------------------------------------------------------------
def _dims(case):
    return [int(d) for d in case["dims"].split("x")]


def _elems(dims):
    """(points, bins of the real transform's half spectrum): its first axis is the halved one."""
    d = [x for x in dims if x != 1] or [1]
    n = math.prod(d)
    return n, (d[0] // 2 + 1) * (n // d[0])


def _steps(case):
    return case["kind"].split("+")


def _mix(case):
    """The queue's transforms: 75% 1D, 20% 2D, 5% 3D, half of them real, half inverse."""
    r = random.Random(case["mix"])
    out = []
    for _ in range(case["count"]):
        u = r.random()
        if u < 0.75:
            dims = [1 << r.randint(6, 18)]
        elif u < 0.95:
            dims = [1 << r.randint(6, 11) for _ in range(2)]
        else:
            dims = [1 << r.randint(5, 8) for _ in range(3)]
        out.append((r.choice(["c", "ci", "r", "ri"]), dims))
    return out


def _sides(kind, dims):
    """Arrays of one transform: (count, elements) in and out, split format."""
    n, h = _elems(dims)
    return {"c": ((2, n), (2, n)), "ci": ((2, n), (2, n)), "r": ((1, n), (2, h)), "ri": ((2, h), (1, n))}[kind]


def _queue_layout(case):
    """Offsets of every transform's arrays in one buffer, inputs first: [(kind, dims, in offsets, out offsets)], input floats, all floats."""
    items, at = [], 0
    for kind, dims in _mix(case):
        count, m = _sides(kind, dims)[0]
        ins = []
        for _ in range(count):
            ins.append(at)
            at += (m + 63) // 64 * 64
        items.append([kind, dims, ins, []])
    inputs = at
    for it in items:
        count, m = _sides(it[0], it[1])[1]
        for _ in range(count):
            it[3].append(at)
            at += (m + 63) // 64 * 64
    return items, inputs, at


# ---------------------------------------------------------------------------
# inputs and plans
# ---------------------------------------------------------------------------
def _normal(shape, bits, seed, dev):
    g = torch.Generator(device=dev)
    g.manual_seed(seed)
    return torch.randn(shape, generator=g, device=dev, dtype=torch.float64 if bits == 64 else torch.float32)


def _input(case, seed, dev):
    """The arrays the first step reads: standard normal, re then im, or re,im pairs, or one real array."""
    n, h = _elems(_dims(case))
    first = _steps(case)[0]
    m = (h if first == "ri" else n) * case["batch"]
    if first == "r":
        return [_normal(m, case["bits"], seed, dev)]
    if case["inter"]:
        return [_normal(2 * m, case["bits"], seed, dev)]
    x = _normal((2, m), case["bits"], seed, dev)
    return [x[0], x[1]]


def _output(case, step, new):
    n, h = _elems(_dims(case))
    m = (h if step == "r" else n) * case["batch"]
    if step == "ri":
        return [new(m)]
    return [new(2 * m)] if case["inter"] else [new(m), new(m)]


_CLASSES = {"c": G.complex_transform, "ci": G.inverse_complex_transform, "r": G.real_transform,
            "ri": G.inverse_real_transform}


def _args(step, case, src, dst):
    """Array arguments of one call, None for the im arrays of paired data (and of the real side of a BatchPlan launch)."""
    launch = case["api"] == "launch"
    a = [src[0], src[1] if len(src) > 1 else None]
    b = [dst[0], dst[1] if len(dst) > 1 else None]
    if launch:
        return a + b
    if step == "r":
        return [a[0]] + b
    if step == "ri":
        return a + [b[0]]
    return a + b


def prepare(case, seed):
    if case["api"] == "queue":
        items, inputs, total = _queue_layout(case)
        buf = torch.empty(total, device="cuda")
        g = torch.Generator(device="cuda")
        g.manual_seed(seed)
        buf.normal_(generator=g)
        base = buf.data_ptr()
        descs = []
        for kind, dims, ins, outs in items:
            p = [base + 4 * o for o in ins] + ([None] if len(ins) == 1 else [])
            p += [base + 4 * o for o in outs] + ([None] if len(outs) == 1 else [])
            descs.append((kind, dims, *p))
        return {"queue": G.Queue(descs), "buf": buf, "out": buf[inputs:]}
    fmt = G.afft_interleaved if case["inter"] else G.afft_split
    dims, bits = _dims(case), case["bits"]
    dtype = torch.float64 if bits == 64 else torch.float32
    host = case["api"] == "host"
    src = _input(case, seed, "cpu" if host else "cuda")
    if host:
        src = [x.numpy() for x in src]
        new = lambda m: np.zeros(m, np.float64 if bits == 64 else np.float32)  # noqa: E731
    else:
        new = lambda m: torch.empty(m, dtype=dtype, device="cuda")  # noqa: E731
    calls, outs = [], []
    for step in _steps(case):
        dst = _output(case, step, new)
        if case["api"] == "launch":
            plan = G.BatchPlan(step, dims, case["batch"], fmt=fmt, form="f64" if bits == 64 else None)
        else:
            plan = _CLASSES[step](dims, fmt=fmt, bits=bits)
        calls.append((plan, _args(step, case, src, dst)))
        outs.append(dst)
        src = dst
    return {"launch": case["api"] == "launch", "calls": calls, "out": outs}


def run(state):
    if "queue" in state:
        state["queue"].run(torch.cuda.current_stream())
    elif state["launch"]:
        stream = torch.cuda.current_stream()
        for plan, args in state["calls"]:
            plan.launch(*args, stream=stream)
    else:
        for plan, args in state["calls"]:
            plan(*args)
    return state["out"]


# ---------------------------------------------------------------------------
# what a pass cannot do without, and its exact result
# ---------------------------------------------------------------------------
def _work(kind, dims, bits):
    (ci, mi), (co, mo) = _sides(kind, dims)
    n = math.prod(dims)
    flops = (5.0 if kind in ("c", "ci") else 2.5) * n * max(1.0, math.log2(n))
    return (ci * mi + co * mo) * (bits // 8), flops


def work(case):
    if case["api"] == "queue":
        each = [_work(kind, dims, 32) for kind, dims in _mix(case)]
        return {"bytes": float(sum(b for b, _ in each)), "flops": float(sum(f for _, f in each))}
    each = [_work(step, _dims(case), case["bits"]) for step in _steps(case)]
    return {"bytes": float(sum(b for b, _ in each)) * case["batch"], "flops": sum(f for _, f in each) * case["batch"]}


def _transform64(kind, dims, z):
    """One step in 64 bits on z, (batch, elements): complex, or real into r.  Inverses are unnormalised; a real transform
    halves its first axis, and its inverse takes only the real parts of the first and the last plane after the other
    axes' inverses."""
    d = [x for x in dims if x != 1] or [1]
    axes = list(range(1, len(d) + 1))
    n = math.prod(d)
    if kind == "c":
        return torch.fft.fftn(z.reshape([-1] + d), dim=axes).reshape(-1, n)
    if kind == "ci":
        return torch.fft.ifftn(z.reshape([-1] + d), dim=axes, norm="forward").reshape(-1, n)
    if kind == "r":
        if n == 1:
            return z.to(torch.complex128)
        full = torch.fft.rfft(z.reshape([-1] + d), dim=1)
        if len(d) > 1:
            full = torch.fft.fftn(full, dim=axes[1:])
        return full.reshape(full.shape[0], -1)
    x = z.reshape([-1, d[0] // 2 + 1] + d[1:])
    if n == 1:
        return x.real.reshape(-1, 1)
    if len(d) > 1:
        x = torch.fft.ifftn(x, dim=axes[1:], norm="forward")
    x = x.clone()
    x[:, 0].imag = 0
    x[:, d[0] // 2].imag = 0
    return torch.fft.irfft(x, n=d[0], dim=1, norm="forward").reshape(-1, n)


def _complex(arrays, inter):
    if inter:
        return torch.view_as_complex(arrays[0].double().reshape(-1, 2))
    return torch.complex(arrays[0].double(), arrays[1].double())


def _arrays(z, inter):
    z = z.reshape(-1)
    if not z.is_complex():
        return [z]
    return [torch.view_as_real(z).reshape(-1)] if inter else [z.real.contiguous(), z.imag.contiguous()]


def exact(case, seed):
    if case["api"] == "queue":
        items, inputs, total = _queue_layout(case)
        buf = torch.empty(total, device="cuda")
        g = torch.Generator(device="cuda")
        g.manual_seed(seed)
        buf.normal_(generator=g)
        out = buf[inputs:].double()
        for kind, dims, ins, outs in items:
            m = _sides(kind, dims)[0][1]
            x = [buf[o:o + m] for o in ins]
            z = x[0].double() if kind == "r" else _complex(x, False)
            for o, y in zip(outs, _arrays(_transform64(kind, dims, z.reshape(1, -1)), False)):
                out[o - inputs:o - inputs + y.numel()] = y
        return out
    host = case["api"] == "host"
    src = [x.cuda() for x in _input(case, seed, "cpu" if host else "cuda")]
    steps = _steps(case)
    z = src[0].double() if steps[0] == "r" else _complex(src, case["inter"])
    z = z.reshape(case["batch"], -1)
    outs = []
    for step in steps:
        z = _transform64(step, _dims(case), z)
        outs.append([a.cpu().numpy() if host else a for a in _arrays(z, case["inter"])])
    return outs
