"""Three passes along an FP64 axis take the scratch of two: the middle one runs
in place on the first one's output."""
import pytest

import fft_gb300 as G
from plan_emulator import describe


@pytest.mark.parametrize("kind,log,batch,fmt", [
    ("c", 20, 8, 0), ("ci", 20, 128, 0), ("c", 22, 2, 1), ("ci", 21, 4, 0), ("c", 20, 100, 1)])
def test_three_passes(kind, log, batch, fmt):
    desc = describe(kind, [1 << log], batch, fmt | G.FORM_F64)
    assert len(desc["ops"]) == 3
    assert desc["scratch_elems"] == 2 * batch << log
    first, middle, last = desc["ops"]
    assert middle["in"] == middle["out"] == dict(middle["in"], **{k: first["out"][k] for k in ("re", "im")})
    assert [last["in"][k] for k in ("re", "im")] == [middle["out"][k] for k in ("re", "im")]
