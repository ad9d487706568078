"""How many temporaries a right-hand side may park.  The rollout records keep a spill slot for every state and
have the rest of the encoder's 48 for themselves: a program whose routine calls hold four shared arguments
on each of six levels fits beside eight states, and scores like the CPU restatement in every lane width."""
import numpy as np
import pytest
import torch

import support as S
from secant_b200 import programs as P
from secant_b200.runner import rk4_score
from test_encoder_cpu import encode, host_eval, info, same

STATES = 8
op, arg = P.op, P.arg


def nested(levels):
    """Routine k combines its four arguments for routine k + 1 and uses each of them again afterwards."""
    half = P.lit(0.5) + op("MUL")
    last = arg(0) + arg(1) + op("MUL") + arg(2) + arg(3) + op("MUL") + op("SUB") + P.RET
    routines = []
    for k in range(levels - 1):
        inner = b"".join(arg(i) + arg((i + 1) % 4) + op("ADD") + half for i in range(4)) + P.routine(k + 1)
        routines.append(inner + arg(0) + op("MUL") + arg(1) + op("ADD") + arg(2) + op("MUL") + arg(3) + op("SUB") + half + P.RET)
    return routines + [last]


def right_hand_sides(levels=7):
    first = lambda s: b"".join(P.col((s + i) % STATES) + P.col((s + i + 1) % STATES) + op("SUB") for i in range(4))  # noqa: E731
    return P.PackedPrograms([first(s) + P.routine(0) + P.col(s) + op("SUB") + P.RET for s in range(STATES)], nested(levels))


def test_temporaries_begin_behind_one_slot_a_state():
    pop = right_hand_sides()
    code, handle = encode(pop, STATES, 0, True, 0, rollout=True)
    assert code == 0
    x = np.stack([P.uniform(3, c, 5, -1, 1) for c in range(STATES)])
    _, want = S.oracle_toggle_materialize(pop, x, np.zeros((1, 1), dtype=np.float32), 0, 0, 0)
    for a in range(STATES):
        assert 24 <= info(handle, a)[1] - STATES <= 40
        assert all(same(host_eval(handle, a, x, None, 0, row), want[a, row]) for row in range(5))
    S.hooks().sbt_free(handle)


@pytest.mark.gpu
@pytest.mark.parametrize("trajectories", [3, 40, 100])
def test_many_temporaries_beside_eight_states(cuda, trajectories):
    points, pop = 5, right_hand_sides()
    times = (np.arange(points, dtype=np.float32) * np.float32(0.05)).astype(np.float32)
    ref = np.stack([P.uniform(31, s, trajectories * points, -1, 1) for s in range(STATES)])
    dev = lambda a: torch.tensor(np.ascontiguousarray(a), device="cuda")  # noqa: E731
    got = rk4_score(pop, STATES, dev(ref), dev(times)).cpu().numpy()[:, 0]
    code, want, want64 = S.oracle_rk4(pop, STATES, ref, trajectories, times, want64=True)
    assert code == 0 and np.isfinite(want).all()
    assert np.allclose(got, want64, rtol=1e-4)      # the same states; only the order of the residual sum differs
