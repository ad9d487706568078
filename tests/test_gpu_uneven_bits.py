"""A program that reads many toggle bits among programs that read few: the same scores whether all constant
tables fit one launch or the programs are cut into launches by their own bits, from host programs and from a
resident population, against the CPU restatement."""
import numpy as np
import pytest
import torch

import support as S
from secant_b200 import abi, programs as P
from secant_b200.runner import Runner

pytestmark = pytest.mark.gpu
BITS, K = 10, 3


def population(few, many):
    """`few` random programs over two bits; `many` that read all bits, at the front, in the middle and at the end."""
    asts = list(P.random_population(41, few, 20, 3, K, 1.0, toggle_bits=2, ops=P.ARITHMETIC_OPS).asts)
    for i in range(many):
        code = P.col(i % 3)
        for b in range(BITS):
            code += P.bank((b + i) % K) + P.col(b % 3) + P.tog2(b) + P.op("ADD") + P.lit(0.5) + P.op("MUL")
        asts.insert(i * few // max(1, many - 1), code + P.RET)
    return P.PackedPrograms(asts)


@pytest.mark.parametrize("few,many,sets,targets", [(40, 1, 1, 1), (400, 3, 5, 1), (60, 2, 12, 2), (0, 4, 2, 1)])
def test_scores_do_not_depend_on_how_the_tables_are_cut(cuda, few, many, sets, targets):
    rows = 97                                                     # one tile: no row splits, so no sum depends on the limit
    rng = np.random.default_rng(few)
    pop = population(few, many)
    x, y = rng.standard_normal((3, rows)).astype(np.float32), rng.standard_normal((targets, rows)).astype(np.float32)
    b = rng.standard_normal((sets, K)).astype(np.float32)
    dev = lambda a: torch.tensor(np.ascontiguousarray(a), device="cuda")  # noqa: E731
    with Runner(abi.SHAPE_TOGGLE_SSE, 3, targets, K, workers=2, streams=2) as rn:
        whole = rn.toggle_sse(pop, dev(x), dev(y), dev(b), sets, BITS).cpu().numpy()
        once = rn.population(pop, BITS)
        for room in (2.5, 1, 0):                                  # tables of that many of the largest programs
            rn.set_scratch_limit(max(4, int(2 * room * 4 * 8 * ((sets + 3) << BITS))))
            cut = rn.toggle_sse(pop, dev(x), dev(y), dev(b), sets, BITS).cpu().numpy()
            assert np.array_equal(cut.view(np.uint32), whole.view(np.uint32)), room
            again = torch.full(whole.shape, -1.0, device="cuda")
            torch.cuda.synchronize()
            once.run(rn.toggle_request(pop, dev(x), dev(y), dev(b), sets, BITS, again))
            assert np.array_equal(again.cpu().numpy().view(np.uint32), whole.view(np.uint32)), room
        once.destroy()
    some = sorted(set(range(0, few + many, max(1, (few + many) // 8))) | {i * few // max(1, many - 1) for i in range(many)})[:12]
    code, _, want64 = S.oracle_toggle_sse(pop.subset(some), x, y, b, K, BITS)
    whole, want64 = whole[some], np.asarray(want64).reshape(whole[some].shape)
    ok = np.isfinite(want64)
    assert code == 0 and ok.mean() > 0.9 and np.allclose(whole[ok], want64[ok], rtol=1e-4, atol=1e-4)
