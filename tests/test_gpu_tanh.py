"""tanh of the evaluator's core around its change of method, at the cut and for every special value: at most
1.5 ulp from float64, odd, and independent of the arguments beside it."""
import numpy as np
import pytest
import torch

from secant_b200 import abi, programs as P
from secant_b200.runner import Runner

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", ["edges", "ordinary", "tiny"])
def test_tanh_against_float64(cuda, kind):
    rng = np.random.default_rng(3)
    if kind == "edges":
        near = np.concatenate([np.float32(l) * (1 + np.arange(-400, 401, dtype=np.float64) * 2.0 ** -23) for l in (0.9, 1.0, 9.0, 10.0)])
        x = np.concatenate([near, [0.0, 1e-45, 1e-38, 88.0, 1e30, 3e38, np.inf, np.nan]]).astype(np.float32)
    elif kind == "ordinary":
        x = rng.uniform(0.0, 10.0, 1 << 18).astype(np.float32)
    else:
        x = np.exp2(rng.uniform(-149, 0, 1 << 16)).astype(np.float32)
    x = np.concatenate([x, -x])
    with Runner(abi.SHAPE_MATERIALIZE, 1, 0) as rn:
        got, again = (rn.materialize(P.PackedPrograms([P.col(0) + P.op("TANH") + P.RET]), torch.tensor(v[None, :], device="cuda")).cpu().numpy()[0]
                      for v in (x, x[::-1].copy()))
    assert np.array_equal(got.view(np.uint32), again[::-1].view(np.uint32))
    want = np.tanh(x.astype(np.float64))
    assert np.array_equal(np.isnan(got), np.isnan(want)) and np.array_equal(np.signbit(got), np.signbit(want))
    ok = ~np.isnan(want)
    assert np.all(np.abs(got[ok] - want[ok]) <= np.maximum(1.5 * np.spacing(np.abs(got[ok])).astype(np.float64), 2.0 ** -149))
