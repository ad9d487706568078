"""What is claimed for every argument, tried for every argument: tanh over all of float32, the approximate
functions inside and outside the evaluator's core over all arguments the core takes, and the sixth of a step
for every significand."""
import numpy as np
import pytest
import torch

from secant_b200 import abi, programs as P
from secant_b200.runner import Runner, rk4_score

pytestmark = pytest.mark.gpu
CHUNK = 1 << 26


def floats(first, last):
    """The float32 numbers of the bit patterns first .. last, in pieces."""
    for at in range(first, last + 1, CHUNK):
        yield torch.arange(at, min(at + CHUNK, last + 1), dtype=torch.int64, device="cuda").to(torch.int32).view(torch.float32)


def bits(a):
    return a.view(torch.int32)


def predict(rn, program, x):
    torch.cuda.synchronize()                                  # the library does not wait for the caller's streams
    return rn.materialize(P.PackedPrograms([program + P.RET]), x if x.ndim == 2 else x[None, :])[0]


def test_tanh_is_within_1_3_ulp_for_every_argument(cuda):
    worst = 0.0
    with Runner(abi.SHAPE_MATERIALIZE, 1, 0) as rn:
        for x in floats(0, 0x7f800000):
            got = predict(rn, P.col(0) + P.op("TANH"), x)
            assert torch.equal(bits(predict(rn, P.col(0) + P.op("TANH"), -x)), bits(-got))
            want = torch.tanh(x.double())
            ulp = torch.ldexp(torch.ones_like(want), torch.clamp(torch.frexp(want).exponent - 24, min=-149))
            worst = max(worst, float(((got.double() - want).abs() / ulp).max()))
    print(f"tanh: at most {worst:.3f} ulp")
    assert worst <= 1.3


# the core's arguments (bit patterns of the magnitudes), one beyond them, and whether both signs belong to them
@pytest.mark.parametrize("name,first,last,outside,signs", [("EXP", 0, 0x42AE0000, 88.5, 2), ("LOG", 0x00800000, 0x7f800000, 1e-40, 1),
                                                           ("DIV", 0x00800000, 0x7E800000, 1e-40, 2)])
def test_approximate_functions_have_the_same_bits_inside_and_outside_the_core(cuda, name, first, last, outside, signs):
    """Every argument once among common ones and once with an unusual one in its group of 128 rows, which sends
    the whole tile out of the core."""
    program = (P.lit(1.7) + P.col(0) if name == "DIV" else P.col(0)) + P.op(name)
    with Runner(abi.SHAPE_MATERIALIZE, 1, 0) as rn:
        rn.set_math(True)
        for magnitudes in floats(first, last):
            for x in (magnitudes, -magnitudes)[:signs]:
                x = torch.nn.functional.pad(x, (0, -x.numel() % 127), value=1.0).view(-1, 127)
                inside, left = (predict(rn, program, torch.nn.functional.pad(x, (0, 1), value=v).view(-1)).view(-1, 128)[:, :127]
                                for v in (1.0, outside))
                assert torch.equal(bits(inside.contiguous()), bits(left.contiguous()))


def test_approximate_quotients_have_the_same_bits_for_any_dividend(cuda):
    g = torch.Generator(device="cuda")
    g.manual_seed(4)
    n = 127 << 18
    pairs = torch.randint(-(1 << 31), 1 << 31, (2, n), generator=g, device="cuda").to(torch.int32).view(torch.float32)
    pairs[1] = torch.where((pairs[1].abs() >= 2.0 ** -126) & (pairs[1].abs() <= 2.0 ** 126), pairs[1], torch.ones_like(pairs[1]))
    program = P.col(0) + P.col(1) + P.op("DIV")
    with Runner(abi.SHAPE_MATERIALIZE, 2, 0) as rn:
        rn.set_math(True)
        inside, left = (predict(rn, program, torch.nn.functional.pad(pairs.view(2, -1, 127), (0, 1), value=v).view(2, -1)).view(-1, 128)[:, :127].contiguous()
                        for v in (1.0, 1e-40))
    same = (bits(inside) == bits(left)) | (inside.isnan() & left.isnan())
    assert bool(same.all()), int((~same).sum())


@pytest.mark.parametrize("steps", ["every significand", "every exponent"])
def test_the_sixth_of_a_step_is_the_rounded_quotient(cuda, steps):
    """One step of slope 2/3, whose weighted sum rounds to 4 exactly: the state is four sixths of the step, and
    the score is zero when every trajectory's is the float32 quotient's."""
    f = np.float32(2 / 3)
    total = f
    for weight in (2, 2, 1):
        total = np.float32(np.float64(weight) * np.float64(f) + np.float64(total))
    assert total == 4
    if steps == "every significand":
        h = np.arange(0x3f800000, 0x40800000, dtype=np.uint32).view(np.float32)                  # [1, 4)
    else:
        h = np.random.default_rng(6).integers(1, 0x7f7fffff, 1 << 18, dtype=np.uint32).view(np.float32)
    n = h.size
    dev = lambda a: torch.tensor(np.ascontiguousarray(a), device="cuda")  # noqa: E731
    times, reference = np.zeros((2, n, 2), dtype=np.float32)
    times[:, 1] = h
    offsets = dev(2 * np.arange(n + 1, dtype=np.int32))
    program = P.PackedPrograms([P.lit(float(f)) + P.RET])

    def score(end):
        reference[:, 1] = end
        return float(rk4_score(program, 1, dev(reference.reshape(1, -1)), dev(times.reshape(-1)), offsets=offsets).item())
    exact = np.float32(4) * (h / np.float32(6))
    assert score(exact) == 0.0
    exact[n // 3] = np.nextafter(exact[n // 3], np.float32(0))                                  # one unit off in one trajectory shows
    if steps == "every significand":
        assert score(exact) > 0.0
