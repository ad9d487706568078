"""Sine, cosine and exponential of any argument, in every register tile: both sides of every limit and every exponent,
beside common arguments, against float64 and against the bits of the other tiles."""
import numpy as np
import pytest
import torch

from secant_b200 import abi, programs as P
from secant_b200.runner import Runner

pytestmark = pytest.mark.gpu
ROWS = 1024 + 77                                                     # whole passes of every tile and a remainder


def arguments(name, spread):
    """Common arguments with unusual ones in every `spread`-th row."""
    rng = np.random.default_rng(spread)
    x = rng.uniform(-80, 80, ROWS).astype(np.float32)
    at = slice(0, ROWS, spread)
    n = x[at].size
    if name == "EXP":
        special = rng.uniform(-110, 95, n)
    else:                                                            # every exponent from 2^11 on, and both sides of 4,096, 2^20 and 2^50
        special = np.exp2(11 + np.arange(n) * (116.99 / max(1, n - 1))) * rng.choice([-1, 1], n)
        special[1::5] = 2.0 ** 20 * (1 + (np.arange(special[1::5].size) - 8) * 2.0 ** -23)
        special[2::5] = 4096.0 * (1 + (np.arange(special[2::5].size) - 8) * 2.0 ** -23)
        special[3::5] = 2.0 ** 50 * (1 + (np.arange(special[3::5].size) - 8) * 2.0 ** -23)
    x[at] = special.astype(np.float32)
    return x


@pytest.mark.parametrize("name", ["SIN", "COS", "EXP"])
@pytest.mark.parametrize("spread", [1, 7, 129, ROWS])
def test_any_argument_in_every_tile(cuda, name, spread):
    x = arguments(name, spread)
    dev = torch.tensor(x[None, :], device="cuda")
    with Runner(abi.SHAPE_MATERIALIZE, 1, 0) as rn:
        got = rn.materialize(P.PackedPrograms([P.col(0) + P.op(name) + P.RET]), dev)
    with np.errstate(all="ignore"):
        want = getattr(np, name.lower())(x.astype(np.float64))
        ulp = np.maximum(np.spacing(np.abs(want).astype(np.float32)).astype(np.float64), 2.0 ** -149)
    values = got.cpu().numpy()[0].astype(np.float64)
    over = want > np.finfo(np.float32).max
    assert np.array_equal(np.isinf(values), over)
    # the float nearest to x * 2/pi, its product with pi/2 and the polynomial: half an ulp of the argument each, at most
    # 1.6 ulp of a result, and at most 1.2 of the sum; the exponential's estimate and products: 2.5
    assert np.all(np.abs(values - want)[~over] <= 2.8 * ulp[~over])
    # a coefficient of one puts the argument into the main part of the tiles of 16 x 1, 8 x 2 and 4 x 4; the loss against
    # the predictions is zero if, and only if, every value has the same bits
    target = torch.where(torch.isinf(got), torch.zeros_like(got), got)
    for banks in (1, 2, 9):
        with Runner(abi.SHAPE_TOGGLE_SSE, 1, 1, 1) as rn:
            pop = P.PackedPrograms([P.col(0) + P.bank(0) + P.op("MUL") + P.op(name) + P.RET])
            keep = dev if name != "EXP" else torch.clamp(dev, max=88.0)
            if name == "EXP":
                with Runner(abi.SHAPE_MATERIALIZE, 1, 0) as other:
                    target = other.materialize(P.PackedPrograms([P.col(0) + P.op(name) + P.RET]), keep)
            assert torch.count_nonzero(rn.toggle_sse(pop, keep, target, torch.ones((banks, 1), device="cuda"), banks, 0)) == 0


@pytest.mark.parametrize("name,infinite", [("SIN", np.nan), ("COS", np.nan), ("EXP", np.inf)])
def test_infinities_and_nan_beside_numbers(cuda, name, infinite):
    x = arguments(name, 3)
    x[5::11], x[6::13], x[7::17] = np.inf, -np.inf, np.nan
    with Runner(abi.SHAPE_MATERIALIZE, 1, 0) as rn:
        dev = lambda a: torch.tensor(np.ascontiguousarray(a[None, :]), device="cuda")  # noqa: E731
        program = P.PackedPrograms([P.col(0) + P.op(name) + P.RET])
        got, rest = rn.materialize(program, dev(x))[0].cpu().numpy(), rn.materialize(program, dev(np.where(np.isfinite(x), x, 1)))[0].cpu().numpy()
    plus, minus, nan = np.isposinf(x), np.isneginf(x), np.isnan(x)
    assert np.array_equal(got[np.isfinite(x)].view(np.uint32), rest[np.isfinite(x)].view(np.uint32))
    assert np.all(np.isnan(got[nan])) and np.array_equal(got[plus], np.full(plus.sum(), infinite, np.float32), equal_nan=True)
    assert np.array_equal(got[minus], np.full(minus.sum(), 0.0 if name == "EXP" else np.nan, np.float32), equal_nan=True)
