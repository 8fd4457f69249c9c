"""Which FP64 axes a plan takes does not depend on the batch: complex lines of
up to 2^22 points, real ones of up to 2^23, whatever their number of passes."""
import pytest

import fft_gb300 as G
from plan_emulator import describe

F = G.FORM_F64


@pytest.mark.parametrize("kind,longest", [("c", 22), ("ci", 22), ("r", 23), ("ri", 23)])
@pytest.mark.parametrize("fmt", [0, 1])
@pytest.mark.parametrize("batch", [1, 2, 4, 16, 32])
def test_longest(kind, longest, fmt, batch):
    for log in range(19, 29):
        if batch << log > 1 << 31:
            continue
        if log <= longest:
            assert describe(kind, [1 << log], batch, fmt | F)["ops"]
        else:
            with pytest.raises(ValueError, match="longer than"):
                describe(kind, [1 << log], batch, fmt | F)
