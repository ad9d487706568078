"""secant_b200_runner_set_scratch_limit over the model of the CUDA runtime: partial sums, predictions and
constant tables of a launch together stay within the limit, growth included; sums that go straight to the
output take none of it; and what cannot fit (the tables of one program, 128 rows of a batch's predictions)
still runs."""
import ctypes as C

import pytest

from secant_b200 import abi, programs as P
from secant_b200.runner import make_recipe
from test_runner_failures_cpu import Harness, fake, state

KIB = 1 << 10


def scratch_of(lib):
    out = (C.c_uint64 * 2)()
    lib.fake_scratch(out)
    return int(out[0]), int(out[1])          # bytes of the largest allocation, launches with split rows


@pytest.fixture()
def lib():
    lib = fake()
    lib.secant_b200_runner_set_scratch_limit.restype, lib.secant_b200_runner_set_scratch_limit.argtypes = (
        abi.EXPORTED["secant_b200_runner_set_scratch_limit"])
    lib.fake_scratch.argtypes = [C.POINTER(C.c_uint64)]
    lib.fake_reset()
    yield lib
    lib.fake_reset()


class GramHarness(Harness):
    """A Gram-statistics request: 300 programs in cohorts of four, 20,000 rows."""
    ROWS, COHORT, F = 20000, 4, 3

    def __init__(self, lib, programs=300):
        self.lib = lib
        self.pop = P.random_population(12, programs, 16, self.F, 0, 1.0, ops=P.ARITHMETIC_OPS)
        self.recipe = make_recipe(abi.SHAPE_GRAM_STATS, self.F, 1, 0, num_kernels=4, asts_per_kernel=self.COHORT)
        width = self.COHORT * (1 + self.COHORT + 1)
        self.sizes = dict(x=self.F * self.ROWS, y=self.ROWS, out=-(-programs // self.COHORT) * width)
        self.buffers = {k: lib.fake_device_buffer(4 * n) for k, n in self.sizes.items()}
        run = abi.init_header(abi.StaticRun(), abi.RUN_VERSION, abi.SHAPE_GRAM_STATS)
        self.pop.fill(run.programs)
        for field, key, ld in (("input", "x", self.ROWS), ("targets", "y", self.ROWS), ("output", "out", width)):
            m = getattr(run, field)
            m.address, m.num_elements, m.leading_dimension = self.buffers[key], self.sizes[key], ld
        run.num_rows, run.num_targets = self.ROWS, 1
        self.run = run
        self.stats = abi.runner_stats()


class LongHarness(Harness):
    """2,500 programs of 20 configurations over 3,000 rows (six tiles, so the rows are split where there is room):
    200 KB of partial sums for each row split, about 1.2 MB of constant tables."""
    ROWS = 3000


class WideHarness(Harness):
    """One tile of rows, 2,048 configurations."""
    ROWS, BANKS = 100, 512


def largest_scratch(lib, h, limit):
    code, r = h.create(workers=1, streams=2)
    assert code == 0 and lib.secant_b200_runner_set_scratch_limit(r, limit) == 0
    lib.fake_reset()
    assert h.execute(r) == 0
    assert state(lib)["violations"] == 0, lib.fake_last_violation()
    result = scratch_of(lib)
    assert lib.secant_cubin_runner_destroy(r) == 0
    h.release()
    return result


@pytest.mark.parametrize("limit", [16 * KIB, 300 * KIB, 1000 * KIB, 1500 * KIB, 6000 * KIB, 1 << 30])
def test_partial_sums_and_tables_together_stay_within_the_limit(lib, limit):
    used, split = largest_scratch(lib, LongHarness(lib, programs=2500), limit)
    assert 0 < used <= limit and split       # the limit is not kept by never splitting the rows


def test_the_tables_of_one_program_are_the_least_a_launch_takes(lib):
    h = LongHarness(lib, programs=40)
    used, split = largest_scratch(lib, h, 4)
    assert used <= 4 * 64 * ((h.BANKS + 3) << h.BITS) and not split


def test_sums_of_unsplit_rows_take_no_scratch(lib):
    """The rows are one tile, so nothing is split and the sums go straight to the output; these programs read
    no coefficient, so there is no table either."""
    h = WideHarness(lib, programs=200)
    h.pop = P.PackedPrograms([P.col(i % 3) + P.col(0) + P.op("ADD") + P.RET for i in range(200)])
    h.pop.fill(h.run.programs)
    assert largest_scratch(lib, h, 0) == (0, 0)


@pytest.mark.parametrize("resident", [False, True])
def test_a_program_with_many_toggle_bits_does_not_size_the_others_tables(lib, resident):
    """600 programs read two bits at most and one reads twelve.  With room for a few tables of its size the
    launches stay few: those of the others are as small as they are alone."""
    class Uneven(Harness):
        ROWS, BITS = 100, 12
    h = Uneven(lib, programs=601)
    asts = list(P.random_population(13, 600, 16, h.F, h.K, 1.0, toggle_bits=2, ops=P.ARITHMETIC_OPS).asts)
    wide = P.col(0) + b"".join(P.bank(b % h.K) + P.col(b % h.F) + P.tog2(b) + P.op("ADD") for b in range(h.BITS))
    h.pop = P.PackedPrograms(asts[:300] + [wide + P.RET] + asts[300:])
    h.pop.fill(h.run.programs)
    code, r = h.create(workers=1, streams=2)
    limit = 8 * 4 * (h.K * (h.BANKS + 3) << h.BITS)
    assert code == 0 and lib.secant_b200_runner_set_scratch_limit(r, limit) == 0
    pop = C.c_void_p()
    if resident:
        assert lib.secant_b200_population_create(r, C.byref(h.run.programs), h.BITS, C.byref(pop)) == 0
    lib.fake_reset()
    assert (lib.secant_b200_population_run(pop, C.byref(h.run), C.byref(h.stats)) if resident else h.execute(r)) == 0
    assert state(lib)["violations"] == 0 and 0 < scratch_of(lib)[0] <= limit
    assert state(lib)["launches"] <= 6, state(lib)
    if resident:
        assert lib.secant_b200_population_destroy(pop) == 0
    assert lib.secant_cubin_runner_destroy(r) == 0
    h.release()


@pytest.mark.parametrize("limit", [400 * KIB, 1000 * KIB, 4000 * KIB])
def test_predictions_and_tables_of_the_gram_shape_stay_within_the_limit(lib, limit):
    used, _ = largest_scratch(lib, GramHarness(lib), limit)
    assert 0 < used <= limit


def test_the_gram_shape_takes_at_least_128_rows(lib):
    used, _ = largest_scratch(lib, GramHarness(lib), 4)
    assert 4 * 128 * 300 <= used <= 4 * (128 * 300 + 4 * 300 * 16)
