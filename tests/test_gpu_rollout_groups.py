"""Groups of warps in the rollout scorer: one warp per state, passes of 32, 64 and 128 trajectories, and
arguments the inlined functions leave to the general ones, against the CPU restatement."""
import numpy as np
import pytest
import torch

import support as S
from secant_b200 import programs as P
from secant_b200.runner import rk4_score

pytestmark = pytest.mark.gpu


def right_hand_sides(num_states):
    """One per form; each damped by its state, none further from the others than one step allows."""
    col, lit, op = P.col, P.lit, P.op
    x, y = (lambda s: col(s)), (lambda s: col((s + 1) % num_states))
    forms = [
        lambda s: x(s) + y(s) + op("MUL") + op("SIN"),
        lambda s: y(s) + lit(5000.0) + op("ADD") + op("SIN"),                                         # beyond the short reduction
        lambda s: y(s) + lit(0.5) + op("MUL") + lit(87.5) + op("ADD") + op("EXP") + lit(1e-38) + op("MUL"),
        lambda s: y(s) + lit(3.0) + op("ADD") + lit(1e-39) + op("MUL") + op("LOG") + lit(90.0) + op("ADD"),
        lambda s: y(s) + lit(1e25) + op("DIV") + lit(1e25) + op("MUL"),
        lambda s: lit(1e25) + y(s) + lit(3.0) + op("ADD") + op("DIV") + lit(1e-25) + op("MUL"),
        lambda s: x(s) + y(s) + lit(2.5) + op("ADD") + op("DIV") + x(s) + op("MIN") + y(s) + op("NEG") + op("MAX") + op("ABS"),
        lambda s: x(s) + y(s) + lit(0.25) + op("FMA") + y(s) + op("COS") + op("MUL") + op("TANH"),
    ]
    return [forms[(s + sys) % len(forms)](s) + col(s) + op("SUB") + P.RET for sys in range(len(forms)) for s in range(num_states)]


@pytest.mark.parametrize("num_states", [1, 2, 3, 5, 8])
@pytest.mark.parametrize("trajectories", [1, 32, 33, 64, 65, 129])
def test_states_and_trajectories_at_the_edges_of_a_pass(cuda, num_states, trajectories):
    points = 3
    pop = P.PackedPrograms(right_hand_sides(num_states))
    times = np.array([0.0, 0.01, 0.03], dtype=np.float32)
    ref = np.stack([P.uniform(21, s, trajectories * points, -1, 1) for s in range(num_states)])
    dev = lambda a: torch.tensor(np.ascontiguousarray(a), device="cuda")  # noqa: E731
    for substeps in (1, 3):
        got = rk4_score(pop, num_states, dev(ref), dev(times), steps_per_observation=substeps).cpu().numpy()[:, 0]
        code, want = S.oracle_rk4(pop, num_states, ref, trajectories, times, substeps=substeps)
        assert code == 0 and np.isfinite(want).all()
        assert np.allclose(got, want, rtol=2e-4, atol=1e-6), (got, want)
