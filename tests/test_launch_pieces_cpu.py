"""Launches of one kind of programs cut into pieces by the scratch limit (csrc/runner.cpp: tables_that_fit, launch_batch),
over the model of the CUDA runtime: what the planner is told of a piece is the piece's own."""
import ctypes as C

import pytest

from secant_b200 import abi, programs as P
from test_runner_failures_cpu import Harness, fake, state

CUT = "stream programs grid tile splits rows parts total_cost max_cost main_cost prelude_cost first".split()


def cuts(lib):
    lib.fake_cuts.restype, lib.fake_cuts.argtypes = C.c_size_t, [C.POINTER(C.c_uint64), C.c_size_t]
    n = lib.fake_cuts(None, 0)
    words = (C.c_uint64 * (n * len(CUT)))()
    lib.fake_cuts(words, n)
    return [dict(zip(CUT, words[i * len(CUT):(i + 1) * len(CUT)])) for i in range(n)]


def deep(levels, i):
    """A balanced tree of coefficients and columns: a spill slot for every level."""
    if levels == 0:
        return P.bank(i % 4) + P.col(i % 3) + P.op("MUL")
    return deep(levels - 1, 2 * i) + deep(levels - 1, 2 * i + 1) + P.op("ADD")


class Pieces(Harness):
    """Light programs that all read the same three toggle bits, and a few with many temporaries."""
    ROWS, BANKS, BITS, K, F = 3000, 5, 3, 4, 3

    def __init__(self, lib, light, heavy):
        super().__init__(lib, programs=light + heavy)
        toggled = P.bank(0) + b"".join(P.bank(1 + b) + P.col(b) + P.tog2(b) + P.op("ADD") for b in range(3))
        # two lengths: the longer ones come first in launch order
        asts = [toggled + (P.bank(0) + P.op("MUL")) * (1 + i % 2) + P.RET for i in range(light)]
        self.pop = P.PackedPrograms(asts + [deep(5, i) + P.RET for i in range(heavy)])
        self.pop.fill(self.run.programs)


def run(lib, h, streams, limit):
    code, r = h.create(workers=1, streams=streams)
    assert code == 0
    lib.secant_b200_runner_set_scratch_limit.restype, lib.secant_b200_runner_set_scratch_limit.argtypes = (
        abi.EXPORTED["secant_b200_runner_set_scratch_limit"])
    assert lib.secant_b200_runner_set_scratch_limit(r, limit) == 0
    lib.fake_reset()
    assert h.execute(r) == 0
    assert state(lib)["violations"] == 0, lib.fake_last_violation()
    got = cuts(lib)
    assert lib.secant_cubin_runner_destroy(r) == 0
    return got


@pytest.fixture()
def lib():
    lib = fake()
    lib.fake_reset()
    yield lib
    lib.fake_reset()


@pytest.mark.parametrize("heavy", [0, 3])
def test_a_piece_has_the_weights_of_its_own_programs(lib, heavy):
    h = Pieces(lib, 300, heavy)
    whole = run(lib, h, 1, 0)
    pieces = run(lib, h, 1, 2 * 4 * 20 * 8 * ((h.BANKS + 3) << h.BITS))
    h.release()
    assert len(pieces) >= len(whole) + 4
    for key in ("programs", "total_cost", "main_cost", "prelude_cost"):
        assert sum(p[key] for p in pieces) == sum(w[key] for w in whole), key
    assert all(p["max_cost"] <= p["total_cost"] <= p["programs"] * p["max_cost"] for p in pieces)


@pytest.mark.parametrize("light,heavy", [(300, 3), (300, 60), (80, 3)])
def test_pieces_on_one_stream_do_not_make_room_for_one_another(lib, light, heavy):
    """A launch leaves room for one on another stream; the pieces of one kind of programs follow each other on theirs, so
    pieces of the same weights are cut alike."""
    h = Pieces(lib, light, heavy)
    pieces = run(lib, h, 2, 2 * 4 * 10 * 8 * ((h.BANKS + 3) << h.BITS))
    h.release()
    assert len({p["stream"] for p in pieces}) == 2
    alike = {}
    for p in pieces:
        alike.setdefault((p["stream"], p["programs"], p["total_cost"]), set()).add((p["grid"], p["splits"], p["tile"], p["rows"], p["parts"]))
    assert len(pieces) > len(alike) and all(len(c) == 1 for c in alike.values()), alike
