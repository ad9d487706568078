"""The pair machine of the evaluator where it can go wrong: division over the whole float32 range against
IEEE division, arguments on both sides of every range limit next to common ones, and every operation on
every operand kind in every register tile against the CPU restatement (bit for bit where the operations
are exactly rounded)."""
import numpy as np
import pytest
import torch

import support as S
from secant_b200 import abi, programs as P
from secant_b200.runner import Runner

pytestmark = pytest.mark.gpu


def dev(a):
    return torch.tensor(np.ascontiguousarray(a), device="cuda")


def predictions(programs, x):
    with Runner(abi.SHAPE_MATERIALIZE, x.shape[0], 0) as rn:
        return rn.materialize(P.PackedPrograms(programs), dev(x)).cpu().numpy()


def same_bits(a, b):
    return np.array_equal(np.isnan(a), np.isnan(b)) and np.array_equal(a.view(np.uint32)[~np.isnan(a)], b.view(np.uint32)[~np.isnan(b)])


@pytest.mark.parametrize("kind", ["ordinary", "any bits", "edges"])
def test_division_is_correctly_rounded(cuda, kind):
    rng = np.random.default_rng(5)
    n = 1 << 20
    if kind == "ordinary":                      # inside the common range: the pair path
        x = (rng.standard_normal((2, n)) * 10.0 ** rng.uniform(-8, 8, (2, n))).astype(np.float32)
        x[0, ::97] = 0.0
        x[0, 1::97] = -0.0
    elif kind == "any bits":
        x = rng.integers(0, 1 << 32, (2, n), dtype=np.uint64).astype(np.uint32).view(np.float32)
    else:                                       # mantissas of few bits, limits of the common range, denormals, zeros, infinities
        base = np.array([1.0, 1.5, np.float32(2) - np.float32(2) ** -23, 1 + 2.0 ** -23], dtype=np.float32)
        scale = np.array([0.0, 2.0 ** -149, 2.0 ** -126, 2.0 ** -61, 2.0 ** -60, 1.0, 2.0 ** 60, 2.0 ** 61, 2.0 ** 127, np.inf, np.nan])
        with np.errstate(over="ignore", invalid="ignore"):
            v = np.concatenate([(base[:, None] * scale).astype(np.float32).ravel(), (-base[:, None] * scale).astype(np.float32).ravel()])
        x = np.stack([np.repeat(v, v.size), np.tile(v, v.size)])
    with np.errstate(all="ignore"):
        want = x[0] / x[1]
    got = predictions([P.col(0) + P.col(1) + P.op("DIV") + P.RET], x)[0]
    assert same_bits(got, want)


@pytest.mark.parametrize("name,limits", [("SIN", (4096.0, 2.0 ** 50)), ("COS", (4096.0, 2.0 ** 50)), ("EXP", (86.0, 89.0, -104.0)),
                                         ("LOG", (2.0 ** -126, 1.0))])
def test_a_value_has_the_same_bits_beside_any_other(cuda, name, limits):
    """A tile of common arguments, and the same arguments with every other row replaced by one the common
    path does not take: what stayed keeps its bits, and both sides of every limit agree with float64."""
    rng = np.random.default_rng(6)
    near = np.concatenate([np.float32(l) * (1 + np.arange(-40, 41, dtype=np.float64) * 2.0 ** -23) for l in limits]).astype(np.float32)
    unusual = np.concatenate([near, -near, np.array([np.inf, -np.inf, np.nan, 0.0, -0.0, 1e-42, 3e38, -3e38, 1e15, 1e25], dtype=np.float32)])
    clean = rng.uniform(0.5, 80.0, 4099).astype(np.float32)
    mixed = clean.copy()
    mixed[1::2] = np.resize(unusual, mixed[1::2].size)
    prog = [P.col(0) + P.op(name) + P.RET]
    a, b = predictions(prog, clean[None, :])[0], predictions(prog, mixed[None, :])[0]
    assert np.array_equal(a[::2].view(np.uint32), b[::2].view(np.uint32))
    with np.errstate(all="ignore"):
        want = getattr(np, name.lower())(mixed.astype(np.float64))
        want32 = want.astype(np.float32)
    assert np.array_equal(np.isnan(b), np.isnan(want32))
    finite = np.isfinite(want32) & np.isfinite(b)
    assert np.array_equal(np.isinf(b) & ~finite, np.isinf(want32) & ~finite)
    tolerance = np.maximum(2.5 * np.spacing(np.abs(want32[finite])).astype(np.float64), 2.0 ** -149)
    assert np.all(np.abs(b[finite].astype(np.float64) - want[finite]) <= tolerance)


@pytest.mark.parametrize("banks", [1, 3, 9], ids=["16x1", "8x2", "4x4"])
def test_every_operation_on_every_operand_kind(cuda, banks):
    """acc (op) X and X (op) acc for a column, a hoisted row value, a coefficient and a parked value."""
    col, bank, op = P.col, P.bank, P.op
    mixed = col(0) + bank(0) + op("MUL")                                    # computed, depends on row and bank
    operands = {"row": col(1), "hoisted": col(1) + col(2) + op("MUL"), "constant": bank(1),
                "parked": col(2) + bank(1) + op("ADD") + op("ABS")}
    programs = []
    for binary in ("ADD", "SUB", "MUL", "DIV", "MIN", "MAX"):
        for x in operands.values():
            programs += [mixed + x + op(binary) + P.RET, x + mixed + op(binary) + P.RET]
    programs += [mixed + x + op("NEG") + op("ABS") + bank(2) + op("FMA") + P.RET for x in operands.values()]
    programs += [x + P.RET for x in operands.values()]
    rows, K = 777, 3
    rng = np.random.default_rng(banks)
    x = rng.uniform(0.5, 2.0, (3, rows)).astype(np.float32)
    y = rng.standard_normal((1, rows)).astype(np.float32)
    table = rng.uniform(-2, 2, (banks, K)).astype(np.float32)
    pop = P.PackedPrograms(programs)
    with Runner(abi.SHAPE_TOGGLE_SSE, 3, 1, K) as rn:
        got = rn.toggle_sse(pop, dev(x), dev(y), dev(table), banks, 0).cpu().numpy()
    code, _, want = S.oracle_toggle_sse(pop, x, y, table, K, 0)
    assert code == 0 and np.allclose(got, want, rtol=3e-6)
