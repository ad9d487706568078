"""The cut of small launches into queue items and CTAs (balance_small, csrc/planner.cpp): whole waves, warps
that fit, every item covered, the tiles and row splits inside the data, and one order of addition for every cut."""
import pytest

from test_planner_cpu import AFFINE, LEAVES, MATERIALIZE, NONE, SHARES, SMEM, SSE, plan


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
    assert p["items"] == -(-programs // p["groups"]) * per_program * p["parts"] < (1 << 32) - 20
    assert p["rows_per_split"] % p["tile_rows"] == 0 and p["rows_per_split"] * (p["splits"] - 1) < rows <= p["rows_per_split"] * p["splits"]
    if 148 < p["grid"] < 8 * 148:                                # a last wave of a few CTAs costs a whole wave
        assert p["grid"] % 148 == 0 or p["grid"] % 148 > 148 - p["splits"] or p["groups"] == programs


def order(p):
    """In which order a launch adds the rows of a sum: the pass, the tile and the split they are of.  Totals of passes are
    added as the rules' cut would add them."""
    return (p["variant"],) + ((p["rule_tile"], p["rule_rows"]) if p["pass_sums"] else (p["tile_rows"], p["rows_per_split"]))


HEAVY = dict(slots=6, table=14)
UNEVEN = (60000, 900, 40000, 9000)


@pytest.mark.parametrize("mode,targets", [(SSE, 1), (SSE, 3), (AFFINE, 2)])
@pytest.mark.parametrize("programs,rows,sets", [(900, 9000, 20), (250, 10007, 20), (400, 20000, 20), (64, 4096, 1), (3000, 20011, 1), (124, 47735, 8),
                                                (488, 5823, 16), (17, 262144, 64), (2000, 20000, 64), (1, 1 << 20, 3), (5, 129, 2)])
@pytest.mark.parametrize("kind", [{}, HEAVY])
@pytest.mark.parametrize("scratch", [1 << 28, 1 << 21])
def test_a_neighbour_decides_about_time_alone(mode, targets, programs, rows, sets, kind, scratch):
    for weights in (None, UNEVEN):
        same = dict(banks=1 if mode == AFFINE else sets, mode=mode, targets=targets, scratch=scratch, weights=weights, **kind)
        seen = set()
        for neighbour, share in [(NONE, 1.0)] + [(k, s) for k in (SHARES, LEAVES) for s in (0.05, 0.3, 0.5, 0.8, 0.95)]:
            code, p = plan(programs, rows, neighbour=neighbour, share=share, **same)
            seen.add(order(p))
            passes = -(-rows // (128, 256, 512)[p["variant"]])
            kept = passes if p["pass_sums"] else p["splits"]
            assert code == 1 and p["partial"] == kept * programs * same["banks"] * (targets + (2 if mode == AFFINE else 0))
            # totals are kept of every pass as soon as an item's sums are not of a tile and a split of the rules
            assert p["pass_sums"] == (p["parts"] > 1 or (p["tile_rows"], p["rows_per_split"]) != (p["rule_tile"], p["rule_rows"]))
            assert p["splits"] == 1 or p["partial"] <= scratch
        assert seen == {order(plan(programs, rows, **same)[1])} and len(seen) == 1


@pytest.mark.parametrize("programs,rows,sets,bits", [(1, 97, 5, 8), (129, 5000, 5, 8), (1000, 2001, 1, 8), (30, 40000, 4, 3)])
def test_launches_with_toggles_keep_the_rules_rows(programs, rows, sets, bits):
    for neighbour, share in [(NONE, 1.0), (SHARES, 0.4), (LEAVES, 0.3)]:
        code, p = plan(programs, rows, banks=sets, bits=bits, neighbour=neighbour, share=share)
        assert code == 1 and not p["pass_sums"] and p["parts"] == 1 and (p["tile_rows"], p["rows_per_split"]) == (p["rule_tile"], p["rule_rows"])


@pytest.mark.parametrize("programs,heavy,rows,sets", [(256, 14, 10007, 33), (500, 20, 1537, 1), (61, 7, 129, 9), (300, 20, 200003, 3)])
def test_two_kinds_of_programs_in_one_launch_add_as_each_would(programs, heavy, rows, sets):
    own = [plan(programs - heavy, rows, banks=sets)[1], plan(heavy, rows, banks=sets, **HEAVY)[1]]
    cuts = [x for p in own for x in (p["rule_tile"], p["rule_rows"])]
    code, p = plan(programs, rows, banks=sets, joint=(programs - heavy, *cuts), **HEAVY)
    assert code == 1 and p["pass_sums"] and (p["rule_tile"], p["rule_rows"]) == tuple(cuts[:2])
    passes = -(-rows // (128, 256, 512)[p["variant"]])
    assert p["partial"] == passes * programs * sets
    # without room for the totals of all passes there is no such launch
    assert plan(programs, rows, banks=sets, joint=(programs - heavy, *cuts), scratch=p["partial"], **HEAVY)[0] == 0
