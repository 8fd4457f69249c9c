"""Complex axes of more than 2^22 points have no matrix twiddle table: every
pass of their plans that multiplies by a longer axis's roots has a kernel that
takes the hi/lo pair in all of its forms."""
import pytest

from plan_emulator import describe

MATRIX_MAX = 1 << 22


@pytest.mark.parametrize("kind,logs", [("c", range(21, 31)), ("ci", range(21, 31)), ("ri", range(22, 32)),
                                       ("r", range(20, 24))])
@pytest.mark.parametrize("fmt", [0, 1])
@pytest.mark.parametrize("batch", [1, 2])
def test_tables(kind, logs, fmt, batch):
    for log in logs:
        if log + batch - 1 > 31:
            continue
        ops = [op for op in describe(kind, [1 << log], batch, fmt)["ops"] if op["type"] == "line"]
        assert any(op["tw_n"] for op in ops)
        for op in ops:
            assert op["tw_n"] <= MATRIX_MAX or (op["hilo"] and op["cols"])
            # t2 k < N: the kernels multiply them in 32 bits
            assert (op["tw_qmask"] + 1) << op["logl"] <= max(op["tw_n"], 1 << op["logl"]) <= 1 << 30


# what takes the matrix alone: the TMA and interleaved-pair passes of shorter
# lines, and the pipelined 1024- and 2048-point passes
@pytest.mark.parametrize("kind,dims,fmt,hilo", [
    ("c", [1 << 16], 0, 1), ("c", [1 << 16], 1, 1), ("c", [1 << 18], 0, 0), ("c", [1 << 18], 1, 0),
    ("c", [1 << 20], 0, 0), ("c", [1 << 23], 0, 1), ("c", [1 << 23], 1, 1)])
def test_first_pass(kind, dims, fmt, hilo):
    op = describe(kind, dims, 1, fmt)["ops"][0]
    assert op["tstore"] == 1 and op["hilo"] == hilo
