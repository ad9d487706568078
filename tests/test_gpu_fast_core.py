"""Approximate functions at the edges of what the core computes itself: the same bits for a common argument
whether or not its tile also holds an unusual one, and both sides of every limit near float64."""
import numpy as np
import pytest
import torch

from secant_b200 import abi, programs as P
from secant_b200.runner import Runner

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("name,common,limits", [
    ("SIN", (-3.0, 3.0), (0.5,)), ("COS", (-3.0, 3.0), (0.5,)), ("EXP", (-80.0, 80.0), (87.0, 88.5, -87.0, -88.5)),
    ("LOG", (2.0, 80.0), (2.0 ** -126, 2.0 ** -120, 3e38)), ("DIV", (0.5, 80.0), (2.0 ** -126, 2.0 ** -120, 2.0 ** 125, 2.0 ** 126))])
def test_fast_functions_at_the_limits_of_the_core(cuda, name, common, limits):
    rng = np.random.default_rng(9)
    near = np.concatenate([np.float32(l) * (1 + np.arange(-40, 41, dtype=np.float64) * 2.0 ** -23) for l in limits]).astype(np.float32)
    clean = rng.uniform(*common, 4099).astype(np.float32)
    mixed = clean.copy()
    mixed[1::2] = np.resize(near, mixed[1::2].size)
    program = (P.lit(1.0) + P.col(0) if name == "DIV" else P.col(0)) + P.op(name) + P.RET
    with Runner(abi.SHAPE_MATERIALIZE, 1, 0) as rn:
        rn.set_math(True)
        a, b = (rn.materialize(P.PackedPrograms([program]), torch.tensor(x[None, :], device="cuda")).cpu().numpy()[0] for x in (clean, mixed))
    assert np.array_equal(a[::2].view(np.uint32), b[::2].view(np.uint32))
    x = mixed.astype(np.float64)
    with np.errstate(all="ignore"):
        want = 1.0 / x if name == "DIV" else getattr(np, name.lower())(x)
    normal = (np.abs(want) < 3.4e38) & (np.abs(want) > 2.0 ** -125)
    scale = 1.0 if name in ("SIN", "COS") else np.abs(want[normal]) if name != "LOG" else np.maximum(1.0, np.abs(want[normal]))
    assert np.all(np.abs(b[normal] - want[normal]) <= 2e-5 * scale)
