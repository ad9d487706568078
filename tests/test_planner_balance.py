"""The cut of small launches into queue items and CTAs (balance_small, csrc/planner.cpp): whole waves, warps
that fit, every item covered, and the tiles and row splits (which the sums depend on) inside the data."""
import pytest

from test_planner_cpu import MATERIALIZE, SMEM, SSE, plan


@pytest.mark.parametrize("programs", [1, 7, 129, 148, 149, 1000])
@pytest.mark.parametrize("rows,banks,bits", [(97, 5, 8), (4096, 1, 0), (2001, 1, 8), (10007, 33, 0), (10007, 64, 0), (65536, 16, 0)])
@pytest.mark.parametrize("mode", [SSE, MATERIALIZE])
def test_small_launches_are_cut_to_whole_waves(programs, rows, banks, bits, mode):
    banks, bits = (1, 0) if mode == MATERIALIZE else (banks, bits)
    code, p = plan(programs, rows, banks=banks, bits=bits, mode=mode, targets=0 if mode == MATERIALIZE else 1)
    assert code == 1 and 1 <= p["warps"] <= 20 and p["smem"] <= SMEM
    assert 1 <= p["groups"] <= programs and p["grid"] == p["groups"] * p["splits"]
    bank_groups = -(-banks // (4, 2, 1)[p["variant"]])
    assert bank_groups % p["gpi"] == 0 and (p["ppi"] == 1 or p["gpi"] == bank_groups) and (1 << bits) % p["ppi"] == 0
    per_program = 1 if mode == MATERIALIZE else bank_groups // p["gpi"] * (1 << bits) // p["ppi"]
    assert p["items"] == -(-programs // p["groups"]) * per_program < (1 << 32) - 20
    assert p["rows_per_split"] % p["tile_rows"] == 0 and p["rows_per_split"] * (p["splits"] - 1) < rows <= p["rows_per_split"] * p["splits"]
    if 148 < p["grid"] < 8 * 148:                                # a last wave of a few CTAs costs a whole wave
        assert p["grid"] % 148 == 0 or p["grid"] % 148 > 148 - p["splits"] or p["groups"] == programs
