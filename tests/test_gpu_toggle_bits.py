"""Programs that read few of a run's toggle bits: every permutation gets its score, whichever bits the
program reads, over one tile and several, one row split and several, every register tile and statistic."""
import numpy as np
import pytest
import torch

import support as S
from secant_b200 import abi, programs as P
from secant_b200.runner import Runner

pytestmark = pytest.mark.gpu
BITS = 6


def population(count):
    """Sums of gated columns over the subsets of bits a program may read: none, one, some, all, four-way ones."""
    col, lit, op, bank = P.col, P.lit, P.op, P.bank
    subsets = [(), (0,), (BITS - 1,), (1, 4), (4, 1), (0, 2, 3, 5), tuple(range(BITS))]
    asts = []
    for i in range(count):
        code = col(i % 3) + bank(i % 2) + op("MUL") if i % 4 else col(0) + op("SIN")
        for k, bit in enumerate(subsets[i % len(subsets)]):
            code += col((i + k) % 3) + lit(0.25 * (k + 1)) + P.tog2(bit) + op("ADD")
        if i % 5 == 3:
            code += lit(0.5) + lit(1.5) + lit(-1.0) + bank(0) + P.tog4(BITS - 1, 2) + op("MUL")
        if i % 6 == 5:                                          # between constants only: the bank part's sites
            code += bank(0) + lit(0.75) + P.tog2(3) + lit(1.0) + lit(2.0) + P.tog2(0) + op("ADD") + op("MUL")
        asts.append(code + P.RET)
    return P.PackedPrograms(asts)


@pytest.mark.parametrize("programs,rows,banks,targets", [(1, 97, 1, 1), (45, 97, 5, 1), (45, 4099, 1, 1), (45, 2500, 3, 2), (7, 150001, 2, 1),
                                                         (300, 700, 40, 1), (3000, 70001, 1, 1)])
def test_every_permutation_gets_its_score(cuda, programs, rows, banks, targets):
    rng = np.random.default_rng(11)
    pop = population(programs)
    x, y = rng.standard_normal((3, rows)).astype(np.float32), rng.standard_normal((targets, rows)).astype(np.float32)
    b = rng.standard_normal((banks, 2)).astype(np.float32)
    dev = lambda a: torch.tensor(np.ascontiguousarray(a), device="cuda")  # noqa: E731
    with Runner(abi.SHAPE_TOGGLE_SSE, 3, targets, 2, workers=2, streams=2) as rn:
        got = rn.toggle_sse(pop, dev(x), dev(y), dev(b), banks, BITS).cpu().numpy()
        once = rn.population(pop, BITS)
        again = torch.full(got.shape, -1.0, device="cuda")
        once.run(rn.toggle_request(pop, dev(x), dev(y), dev(b), banks, BITS, again))
        assert np.array_equal(again.cpu().numpy().view(np.uint32), got.view(np.uint32))
        once.destroy()
    few = min(programs, 35)                                     # the subsets and the other forms repeat
    code, _, want64 = S.oracle_toggle_sse(pop.subset(range(few)), x, y, b, 2, BITS)
    assert code == 0 and np.allclose(got[:few], np.asarray(want64).reshape(got[:few].shape), rtol=1e-4, atol=1e-4)
