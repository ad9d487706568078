"""The functions of the rollout machine's core, bit for bit those of the population evaluator's.

A state that starts at zero is integrated over one step of a constant slope f(c), so its value, and with it
the score, is a fixed chain of roundings of f(c), which `score_of` repeats.  A score that is one unit in the
last place of f(c) off is another score for most arguments (checked on the CPU), so a wrong constant in one
of the two machines shows."""
import numpy as np
import pytest
import torch

from secant_b200 import abi, programs as P
from secant_b200.runner import Runner, rk4_score


def score_of(slope, h):
    """Mean squared error of (h / 6 * (f + 2 f + 2 f + f), 0) against (0, 0), every operation rounded to float32."""
    f = slope.astype(np.float64)
    total = f.astype(np.float32)
    for weight in (2.0, 2.0, 1.0):
        total = (weight * f + total).astype(np.float32)
    sixth = np.float32(h) / np.float32(6)
    state = (np.float64(sixth) * total.astype(np.float64)).astype(np.float32)
    return (state.astype(np.float64) ** 2).astype(np.float32) / np.float32(2)


# name, arguments on a linear or a logarithmic scale, signs, step (a power of two that keeps the squares in range)
CASES = [("SIN", (0.01, 4090.0, True), -1, 1.0), ("COS", (0.01, 4090.0, True), -1, 1.0), ("EXP", (1e-3, 40.0, True), -1, 1.0),
         ("EXP", (40.0, 85.9, False), 1, 2.0 ** -64), ("EXP", (40.0, 85.9, False), -2, 2.0 ** 80), ("LOG", (1.2e-38, 3e38, True), 1, 1.0),
         ("LOG", (0.5, 2.0, False), 1, 1.0), ("TANH", (1e-6, 12.0, True), -1, 1.0), ("DIV", (1e-6, 1e6, True), -1, 1.0)]


def arguments(spread, sign, n=6000):
    lo, hi, logarithmic = spread
    rng = np.random.default_rng(17)
    x = np.exp(rng.uniform(np.log(lo), np.log(hi), n)) if logarithmic else rng.uniform(lo, hi, n)
    if sign == -1:
        x[::2] *= -1
    return (-x if sign == -2 else x).astype(np.float32)


@pytest.mark.parametrize("case", CASES, ids=lambda c: f"{c[0]}{c[2]}")
def test_one_unit_in_the_last_place_is_another_score(case):
    name, spread, sign, h = case
    x = arguments(spread, sign).astype(np.float64)
    f = (1.7 / x if name == "DIV" else getattr(np, name.lower())(x)).astype(np.float32)
    off = np.nextafter(f, np.float32(np.inf))
    assert np.all(score_of(f, h) > 0) and np.all(np.isfinite(score_of(f, h)))
    assert np.mean(score_of(f, h) != score_of(off, h)) > 0.6


@pytest.mark.gpu
@pytest.mark.parametrize("trajectories,observed", [(20, 0), (20, 17), (40, 1), (64, 62), (100, 2), (130, 129)])
def test_the_rollout_core_computes_the_evaluators_bits(cuda, trajectories, observed):
    dev = lambda a: torch.tensor(np.ascontiguousarray(a), device="cuda")  # noqa: E731
    op = P.op
    arg = P.col(1) + P.bank(0) + op("ADD")                    # state 1 stays zero: the coefficient itself, in the main part
    offsets = dev((2 * np.arange(trajectories + 1)).astype(np.int32))
    reference = np.zeros((2, trajectories, 2), dtype=np.float32)
    reference[:, :, 1] = np.nan                               # unobserved, except one trajectory's end
    reference[:, observed, 1] = 0.0
    with Runner(abi.SHAPE_MATERIALIZE, 1, 0) as rn:
        for name, spread, sign, h in CASES:
            x = arguments(spread, sign)
            if name == "DIV":                                 # with the computed value above and below the line
                sides = [P.lit(1.7) + arg + op("DIV"), arg + P.lit(1.7) + op("DIV")]
                rows = [P.lit(1.7) + P.col(0) + op("DIV"), P.col(0) + P.lit(1.7) + op("DIV")]
            else:
                sides, rows = [arg + op(name)], [P.col(0) + op(name)]
            for side, row in zip(sides, rows):
                slope = rn.materialize(P.PackedPrograms([row + P.RET]), dev(x[None, :])).cpu().numpy()[0]
                times = np.tile(np.array([0.0, h], dtype=np.float32), trajectories)
                got = rk4_score(P.PackedPrograms([side + P.RET, P.lit(0.0) + P.RET]), 2, dev(reference.reshape(2, -1)), dev(times),
                                dev(x.reshape(1, -1, 1)), 1, x.size, offsets=offsets, allow_missing=True).cpu().numpy()[0]
                want = score_of(slope, h)
                assert np.array_equal(got.view(np.uint32), want.view(np.uint32)), (name, spread, int(np.sum(got != want)))
