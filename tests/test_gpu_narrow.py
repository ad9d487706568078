"""What is the same for all coefficient sets is computed in one bank column of the 4 x 4 tile: functions in row preludes and in
programs without coefficients, common and unusual arguments, chained so that what the other columns hold would show."""
import numpy as np
import pytest
import torch

from secant_b200 import abi, programs as P
from secant_b200.runner import Runner

pytestmark = pytest.mark.gpu
col, bank, lit, op = P.col, P.bank, P.lit, P.op


def expressions():
    x, y = col(0), col(1)
    chain = [x + op("SIN"), x + op("EXP") + op("COS"), x + y + op("MUL") + op("EXP") + op("EXP") + op("SIN"), x + op("ABS") + lit(0.5) + op("ADD") + op("LOG"),
             x + y + op("DIV"), x + op("COS") + y + op("SIN") + op("DIV"), y + x + op("EXP") + op("DIV") + op("TANH"),
             x + op("SIN") + y + op("COS") + op("MUL") + x + op("EXP") + y + op("ABS") + lit(1.0) + op("ADD") + op("LOG") + op("SUB") + op("DIV"),
             lit(3.0) + x + op("SIN") + op("DIV") + op("TANH"), x + op("SIN") + op("SIN") + op("SIN") + op("EXP") + op("LOG")]
    return chain


@pytest.mark.parametrize("fast", [False, True])
@pytest.mark.parametrize("unusual", [0, 3, 200])
@pytest.mark.parametrize("banks", [5, 33])
def test_one_column_serves_all(cuda, fast, unusual, banks):
    """The loss of a prediction against itself is zero for every set, alone (a program without coefficients) and times a
    coefficient of one (a row prelude); its bits are those of the tile of sixteen rows."""
    rows = 1024 + 131
    rng = np.random.default_rng(4)
    x = rng.uniform(-3, 3, (2, rows)).astype(np.float32)
    if unusual:
        x[:, ::unusual] = rng.choice([0.0, 5e6, -2e20, 90.0, -100.0, 1e-40, 3e-39], x[:, ::unusual].shape).astype(np.float32)
    data = torch.tensor(x, device="cuda")
    asts = expressions()
    with Runner(abi.SHAPE_MATERIALIZE, 2, 0) as rn:
        rn.set_math(fast)
        want = rn.materialize(P.PackedPrograms([a + P.RET for a in asts]), data)
    with Runner(abi.SHAPE_TOGGLE_SSE, 2, 1, 1) as rn:
        rn.set_math(fast)
        table = torch.ones((banks, 1), device="cuda")
        for i, a in enumerate(asts):
            rows_here = torch.isfinite(want[i])                    # others have no loss: leave them out
            pop = P.PackedPrograms([a + P.RET, a + bank(0) + op("MUL") + P.RET, a + bank(0) + op("MUL") + a + op("ADD") + a + op("SUB") + P.RET])
            target = want[i][rows_here][None, :].contiguous()
            got = rn.toggle_sse(pop, data[:, rows_here].contiguous(), target, table, banks, 0).reshape(3, banks)
            assert torch.count_nonzero(got[:2]) == 0, i
            assert bool((got[2] <= float((target.double() ** 2).sum()) * 2.0 ** -44 + 1e-30).all()), i    # p + p - p: two roundings of 2^-24
