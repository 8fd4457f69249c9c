"""The FP64 kernels read some lines of a tile after they have stored others (the
lines that fixed point leaves to the FP64 body), so a launch over one buffer
maps each line onto itself: in the plans' own passes in place, and in complex
transforms whose caller's arrays are in place."""
import pytest

import fft_gb300 as G
from plan_emulator import describe

SHAPES = [[8], [64], [4096], [8192], [1 << 14], [1 << 17], [1 << 20], [16, 8], [256, 256], [2048, 64], [8192, 16],
          [64, 32, 16], [2, 2, 2], [128, 8192], [4, 1 << 14]]
DST_RE, DST_IM = 2, 3


def arrays(op, side, in_place):
    """(buffer, first, last) of the elements of a launch's re and im arrays."""
    w, last = op[side], op["nlines"] - 1
    far = (last >> w["qshift"]) * w["hi"] + min(last, w["qmask"]) * w["lo"] + ((1 << op["logl"]) - 1) * w["es"]
    return [(buf - DST_RE if in_place and buf in (DST_RE, DST_IM) else buf, off, off + far)
            for buf, off in (w["re"], w["im"])]


@pytest.mark.parametrize("kind", ["c", "ci", "r", "ri"])
@pytest.mark.parametrize("fmt", [0, 1])
@pytest.mark.parametrize("batch", [1, 8])
def test_lines_map_onto_themselves(kind, fmt, batch):
    for dims in SHAPES:
        for op in describe(kind, dims, batch, fmt | G.FORM_F64)["ops"]:
            if op["type"] != "line" or op["logl"] < 3:
                continue
            src, dst = (arrays(op, side, kind in ("c", "ci")) for side in ("in", "out"))
            if any(a[0] == b[0] and a[1] <= b[2] and b[1] <= a[2] for a in src for b in dst):
                same = dict(op["in"], re=0, im=0) == dict(op["out"], re=0, im=0)
                assert src == dst and same and op["tstore"] == 0, (dims, op)
