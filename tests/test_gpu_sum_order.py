"""One order of addition for a request, however its launches are cut: the same bits for every number of streams, as an entry
among others, from a resident population, and where the scratch leaves only room for the partial sums of the planner's own
row splits."""
import numpy as np
import pytest
import torch

from secant_b200 import abi, programs as P
from secant_b200.runner import Runner

pytestmark = pytest.mark.gpu
SLOTS = 6


def dev(a):
    return torch.tensor(np.ascontiguousarray(a), device="cuda")


def bits(t):
    return t.cpu().numpy().view(np.uint32).copy()


def data(rows, targets, features, seed):
    rng = np.random.default_rng(seed)
    return dev(rng.uniform(-2, 2, (features, rows)).astype(np.float32)), dev(rng.standard_normal((targets, rows)).astype(np.float32))


def tree(levels, i, features, slots):
    """A balanced tree over products: a temporary for every level, which makes it a heavy program from four on."""
    if levels == 0:
        return P.col(i % features) + (P.bank(i % slots) if slots else P.lit(0.5 + 0.25 * (i % 3))) + P.op("MUL")
    sides = tree(levels - 1, 2 * i, features, slots) + tree(levels - 1, 2 * i + 1, features, slots)
    return sides + P.op("ADD" if (levels + i) % 3 else "MUL")


def population(programs, heavy, features, slots, seed):
    """Random programs, and `heavy` that need four to seven temporaries."""
    asts = list(P.random_population(seed, programs - heavy, 24, features, slots, 1.0).asts)
    asts += [tree(4 + i % 4 if heavy > 10 else 4, i, features, slots) + P.RET for i in range(heavy)]
    return P.PackedPrograms(asts, P.PROTECTED_ROUTINES)


def limits(programs, rows, width, rows_of_a_pass):
    """0: no limit of the caller's.  The other is less than the total of every pass takes and more than the splits of tiles of
    four passes and more do, constant tables included."""
    return 0, 4 * int(0.6 * -(-rows // rows_of_a_pass) * programs * width)


@pytest.mark.parametrize("programs,heavy,rows,sets,targets", [(900, 40, 9000, 20, 1), (250, 10, 10007, 20, 1), (400, 30, 20000, 20, 1),
                                                             (120, 120, 30011, 33, 1), (61, 5, 20021, 9, 2), (300, 20, 40009, 3, 1),
                                                             (5, 0, 100003, 64, 1)])
def test_scores_have_the_bits_of_one_order(cuda, programs, heavy, rows, sets, targets):
    pop = population(programs, heavy, 8, SLOTS, programs)
    x, y = data(rows, targets, 8, rows)
    b = dev(np.random.default_rng(1).standard_normal((sets, SLOTS)).astype(np.float32))
    x2, y2 = data(777, targets, 8, 5)
    out, other = torch.empty((programs, targets, sets), device="cuda"), torch.empty((programs, targets, sets), device="cuda")
    got = {}
    for streams in (2, 1, 3):
        for limit in limits(programs, rows, targets * sets, 256 if sets <= 4 else 128):
            with Runner(abi.SHAPE_TOGGLE_SSE, 8, targets, SLOTS, workers=2, streams=streams) as rn:
                rn.set_scratch_limit(limit)
                request = rn.toggle_request(pop, x, y, b, sets, 0, out)
                beside = rn.toggle_request(pop, x2, y2, b, sets, 0, other)
                resident = rn.population(pop, 0)
                calls = {"alone": lambda: rn.run(request), "first": lambda: rn.run_batch([request, beside]),
                         "second": lambda: rn.run_batch([beside, request]), "resident": lambda: resident.run(request)}
                for name, call in calls.items():
                    out.fill_(-1.0)
                    torch.cuda.synchronize()
                    call()
                    got[streams, limit, name] = bits(out)
                resident.destroy()
    first = next(iter(got.values()))
    assert [k for k, v in got.items() if not np.array_equal(v, first)] == []


@pytest.mark.parametrize("shape", [abi.SHAPE_SSE, abi.SHAPE_AFFINE_STATS])
@pytest.mark.parametrize("programs,heavy,rows", [(64, 0, 4096), (500, 30, 20011), (3000, 200, 9001), (7, 2, 300007)])
def test_statistics_have_the_bits_of_one_order(cuda, shape, programs, heavy, rows):
    affine = shape == abi.SHAPE_AFFINE_STATS
    pop = population(programs, heavy, 5, 0, programs)
    x, y = data(rows, 2 if affine else 1, 5, rows)
    width = 4 if affine else 1
    out = torch.empty((programs, width), device="cuda")
    got = {}
    for streams in (2, 1, 3):
        for limit in limits(programs, rows, width, 512):
            with Runner(shape, 5, 2 if affine else 1, workers=2, streams=streams) as rn:
                rn.set_scratch_limit(limit)
                request, resident = rn.static_request(pop, x, y, out), rn.population(pop, 0)
                for name, call in (("alone", rn.run), ("resident", resident.run)):
                    out.fill_(-1.0)
                    torch.cuda.synchronize()
                    call(request)
                    got[streams, limit, name] = bits(out)
                resident.destroy()
    first = next(iter(got.values()))
    assert [k for k, v in got.items() if not np.array_equal(v, first)] == []
