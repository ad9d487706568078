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


@pytest.mark.parametrize("num_states,bits", [(1, 1), (2, 2), (3, 6)])
def test_configurations_share_what_a_system_does_not_read(cuda, num_states, bits):
    """Systems that read no, the lowest, the highest or all toggle bits (in one state or in several): a score for
    every configuration, and the counter as if each had been integrated."""
    col, lit, op, points, trajectories = P.col, P.lit, P.op, 4, 33
    subsets = [(), (0,), (bits - 1,), tuple(range(bits))]
    programs = []
    for i in range(4 * num_states):
        system, s = divmod(i, num_states)
        code = col(s) + P.bank(0) + op("MUL")
        for k, bit in enumerate(subsets[system]):
            if k % num_states == s:
                code += lit(0.1 * (bit + 1)) + col(0) + P.tog2(bit) + op("SUB")
        programs.append(code + op("SIN") + P.RET)
    pop = P.PackedPrograms(programs)
    times = (np.arange(points, dtype=np.float32) * np.float32(0.05)).astype(np.float32)
    ref = np.stack([P.uniform(22, s, trajectories * points, -1, 1) for s in range(num_states)])
    banks = P.normal(23, 0, 8).reshape(4, 2, 1)
    dev = lambda a: torch.tensor(np.ascontiguousarray(a), device="cuda")  # noqa: E731
    counter = torch.zeros(1, dtype=torch.int64, device="cuda")
    got = rk4_score(pop, num_states, dev(ref), dev(times), dev(banks), 1, 2, bits, integrated=counter).cpu().numpy()
    assert int(counter.item()) == 4 * (2 << bits) * trajectories * (points - 1)
    for cfg in range(2 << bits):
        code, want = S.oracle_rk4(pop, num_states, ref, trajectories, times, np.ascontiguousarray(banks[:, cfg >> bits, :]), 1, bits,
                                  cfg & ((1 << bits) - 1))
        assert code == 0 and np.allclose(got[:, cfg], want, rtol=2e-4, atol=1e-6), cfg
