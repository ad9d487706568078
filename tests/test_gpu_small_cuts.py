"""Small launches: tiles cut into parts, and programs with many temporaries in one launch with the others.  Every score,
statistic and prediction against the CPU restatement, at row counts around passes, tiles and parts."""
import numpy as np
import pytest
import torch

import support as S
from secant_b200 import abi, programs as P
from secant_b200.runner import Runner

pytestmark = pytest.mark.gpu


def tree(depth, i, constants):
    """A balanced tree over products: a spill slot for every level, which makes it a heavy program from depth four on."""
    if depth == 0:
        return P.col(i % 3) + (P.bank(i % 2) if constants else P.lit(0.5 + 0.25 * (i % 3))) + P.op("MUL")
    return tree(depth - 1, 2 * i, constants) + tree(depth - 1, 2 * i + 1, constants) + P.op("ADD" if (depth + i) % 2 else "MUL")


def population(programs, heavy, constants):
    """`heavy` programs with spill slots among light ones of several lengths."""
    at = set(np.linspace(0, programs - 1, heavy).astype(int).tolist())
    asts = [tree(5, i, constants) + P.RET if i in at else tree(i % 3, i, constants) + P.col(i % 3) + P.op("SUB") + P.RET for i in range(programs)]
    return P.PackedPrograms(asts)


def data(rows, targets, seed=3):
    rng = np.random.default_rng(seed)
    return rng.uniform(-1, 1, (3, rows)).astype(np.float32), rng.standard_normal((targets, rows)).astype(np.float32)


def dev(a):
    return torch.tensor(np.ascontiguousarray(a), device="cuda")


@pytest.mark.parametrize("programs,heavy", [(1, 0), (1, 1), (40, 1), (61, 7), (300, 20)])
@pytest.mark.parametrize("rows", [1, 129, 1025, 10007])
@pytest.mark.parametrize("banks", [1, 3, 9, 33])
def test_scores(cuda, programs, heavy, rows, banks):
    pop = population(programs, heavy, True)
    x, y = data(rows, 1)
    table = np.random.default_rng(5).standard_normal((banks, 2)).astype(np.float32)
    with Runner(abi.SHAPE_TOGGLE_SSE, 3, 1, 2, workers=2, streams=2) as rn:
        out = torch.full((programs, 1, banks), -1.0, device="cuda")
        keep = dev(x), dev(y), dev(table)
        request = rn.toggle_request(pop, *keep, banks, 0, out)
        got = []
        for limit in (0, 4 * 16 * (banks + 3) * 4, 4):                 # all at once; tables of a few programs a launch; one program a launch
            rn.set_scratch_limit(limit)
            torch.cuda.synchronize()
            rn.run(request)
            got.append(out.cpu().numpy().reshape(programs, banks))
            out.fill_(-1.0)
        rn.set_scratch_limit(0)
        torch.cuda.synchronize()
        rn.run(request)
        again = out.cpu().numpy().reshape(programs, banks)
    code, _, want = S.oracle_toggle_sse(pop, x, y, table, 2, 0)
    want = np.asarray(want).reshape(programs, banks)
    # values have the oracle's bits (sums and products); a sum of squares is at most rows / 32 + 20 roundings deep
    bound = (rows / 32 + 20) * 2.0 ** -24
    assert code == 0 and all(np.all(np.abs(g - want) <= bound * np.abs(want)) for g in got)
    assert np.array_equal(again.view(np.uint32), got[0].view(np.uint32))


@pytest.mark.parametrize("programs,heavy", [(1, 1), (61, 7), (500, 20)])
@pytest.mark.parametrize("rows", [1, 511, 1537, 20011])
def test_predictions_and_statistics(cuda, programs, heavy, rows):
    pop = population(programs, heavy, False)
    x, y = data(rows, 2)
    code, want = S.oracle_materialize(pop, x)
    with Runner(abi.SHAPE_MATERIALIZE, 3, 0) as rn:
        assert code == 0 and np.array_equal(rn.materialize(pop, dev(x)).cpu().numpy().view(np.uint32), want.view(np.uint32))
    p = want.astype(np.float64)
    exact = np.stack([p.sum(1), (p * p).sum(1), p @ y[0], p @ y[1]], axis=1)
    size = np.stack([np.abs(p).sum(1), (p * p).sum(1), np.abs(p) @ np.abs(y[0]), np.abs(p) @ np.abs(y[1])], axis=1)
    with Runner(abi.SHAPE_AFFINE_STATS, 3, 2, workers=2, streams=2) as rn:
        out = torch.zeros((programs, 4), device="cuda")
        keep = dev(x), dev(y)
        torch.cuda.synchronize()
        rn.run(rn.static_request(pop, *keep, out))
        assert np.all(np.abs(out.cpu().numpy() - exact) <= (rows / 32 + 20) * 2.0 ** -24 * size + 1e-30)
