"""Right-hand sides by what they begin with: the end of a stage loads a constant or a state itself and goes on with
the second instruction; a fused multiply-add of three operands is started like any other instruction.

Only exactly rounded operations, so the integrated states have the host's bits, and the sums of n non-negative
float32 terms differ from the float64 ones by n * 2^-24 at most."""
import numpy as np
import pytest
import torch

import support as S
from secant_b200 import programs as P
from secant_b200.runner import rk4_score

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("num_states", [1, 2, 3])
@pytest.mark.parametrize("trajectories", [1, 32, 33, 64, 65, 130])
def test_every_beginning_of_a_right_hand_side(cuda, num_states, trajectories):
    col, lit, bank, op = P.col, P.lit, P.bank, P.op
    forms = [
        lambda s: col(s),                                                       # a load alone
        lambda s: bank(0),
        lambda s: lit(0.5) + col(s) + op("SUB"),                                # a constant first
        lambda s: bank(1) + lit(2.0) + op("MUL") + col(s) + op("MUL"),          # a value of the bank part
        lambda s: col(num_states - 1) + bank(0) + op("MUL") + col(s) + op("SUB"),
        lambda s: col(s) + bank(1) + lit(0.25) + op("FMA"),                     # three operands, no accumulator yet
        lambda s: col(s) + col(0) + op("ADD") + col(num_states - 1) + bank(0) + op("ADD") + op("MUL"),  # a temporary besides
    ]
    pop = P.PackedPrograms([forms[(system + s) % len(forms)](s) + P.RET for system in range(len(forms)) for s in range(num_states)])
    points = 4
    times = np.array([0.0, 0.01, 0.03, 0.04], dtype=np.float32)
    ref = np.stack([P.uniform(31, s, trajectories * points, -1, 1) for s in range(num_states)])
    banks = P.uniform(32, 0, 2 * len(forms) * 2, -1, 1).reshape(len(forms), 2, 2)  # systems, sets, slots
    dev = lambda a: torch.tensor(np.ascontiguousarray(a), device="cuda")  # noqa: E731
    for substeps in (1, 3):
        got = rk4_score(pop, num_states, dev(ref), dev(times), dev(banks), 2, 2, steps_per_observation=substeps).cpu().numpy()
        for k in range(2):
            code, _, want = S.oracle_rk4(pop, num_states, ref, trajectories, times, np.ascontiguousarray(banks[:, k, :]), substeps, want64=True)
            assert code == 0 and np.isfinite(want).all()
            assert np.allclose(got[:, k], want, rtol=trajectories * points * num_states * 2.0 ** -24 + 2.0 ** -22, atol=0), (got[:, k], want)
