"""Fused binary blocks against the CPU oracle: per-level sets and parents for every fusing rule
(& | U of one split, & | alone, none), every left tile, and trace counts around a warp's chunk
width (32 lanes x 2 words), where the last chunk is ragged."""
import numpy as np
import pytest

import oracle as O
from ltlb200 import api, gen
from helpers import row_set

pytestmark = pytest.mark.gpu

RULES = {"and_or_until": ((1,) * 8, 6), "and_or": ((1, 2, 1, 1, 2, 3, 3, 2), 6), "single": ((2, 1, 3, 2, 1, 1, 2, 3), 9)}


@pytest.mark.parametrize("tile", [2, 4, 8])
@pytest.mark.parametrize("rule", sorted(RULES))
def test_fused_levels_match_oracle(rule, tile):
    costs, max_cost = RULES[rule]
    with api.Engine(slots_log2=18, cache_bytes=256 << 20, max_rows=1 << 17, left_tile=tile) as eng:
        for npos, nneg in ((1, 1), (30, 33), (32, 32), (64, 65), (100, 93)):
            inst = gen.generate(npos + tile, 3, npos, nneg, 4, 63, 0.5, 5)
            res = eng.learn(inst, costs=costs, max_cost=max_cost, stop_at_found=False, neg_type=1)
            ref = O.learn(inst, costs=costs, max_cost=max_cost, stop_at_found=False, neg_type=1, cache_rows=1 << 17)
            assert (res.device_flags, res.all_ltls) == (0, ref.all_ltls)
            starts = eng.level_starts(max_cost + 2)
            rows, par = eng.read_rows(0, starts[max_cost + 1])
            mask = (np.uint64(1) << inst.lengths.astype(np.uint64)) - np.uint64(1)
            for c in range(costs[0], max_cost + 1):
                assert row_set(rows[starts[c]:starts[c + 1]]) == row_set(ref.level_rows(c)), (npos, nneg, c)
            for r in range(len(inst.alphabet), len(rows)):
                p = int(par[r])
                op, a, b = (p >> 60) & 7, (p >> 30) & 0x3FFFFFFF, p & 0x3FFFFFFF
                assert np.array_equal(O.apply_op(op, rows[a], rows[b] if op in (1, 2, 6) else None, mask)[0], rows[r])


# Operator costs on both sides of each condition under which a candidate is known to be a duplicate from
# its operands' parents (| against & and ~ together, F against G, ~ of letters only); the rule is used on rows of
# 512 words and more.
KNOWN = [((1, 1, 1, 1, 1, 1, 1, 1), 1, 7), ((1, 1, 1, 1, 1, 1, 1, 1), 2, 7), ((1, 1, 1, 3, 1, 1, 1, 2), 1, 8),
         ((1, 1, 3, 1, 1, 1, 1, 2), 1, 8), ((1, 1, 1, 1, 1, 3, 1, 1), 1, 7), ((1, 1, 1, 1, 1, 1, 3, 1), 1, 7),
         ((1, 2, 2, 2, 1, 1, 1, 1), 1, 8), ((2, 1, 1, 1, 1, 1, 1, 1), 1, 10), ((1, 1, 2, 2, 3, 1, 2, 2), 1, 9)]


@pytest.mark.parametrize("costs,neg,max_cost", KNOWN)
def test_known_duplicates_lose_no_set(costs, neg, max_cost):
    """Every level's set and per-block counts are the oracle's, on long random traces (few accidental
    duplicates) and on short ones (many)."""
    with api.Engine(slots_log2=20, cache_bytes=512 << 20, max_rows=1 << 18) as eng:
        for props, n, lmin, lmax in ((2, 520, 16, 40), (3, 514, 3, 7), (1, 600, 8, 30)):
            inst = gen.generate(props + n, props, n // 2, n // 2, lmin, lmax, 0.5, 4)
            for schedule in (api.SCHEDULE_FUSED, api.SCHEDULE_PER_BLOCK):
                mc = max_cost - (2 if props == 3 or schedule == api.SCHEDULE_PER_BLOCK else 0)
                res = eng.learn(inst, costs=costs, max_cost=mc, stop_at_found=False, neg_type=neg, schedule=schedule)
                ref = O.learn(inst, costs=costs, max_cost=mc, stop_at_found=False, neg_type=neg, cache_rows=1 << 18)
                assert (res.device_flags, res.all_ltls, res.rows) == (0, ref.all_ltls, ref.num_rows)
                starts = eng.level_starts(mc + 2)
                rows, _ = eng.read_rows(0, starts[mc + 1])
                for c in range(costs[0], mc + 1):
                    assert row_set(rows[starts[c]:starts[c + 1]]) == row_set(ref.level_rows(c)), (props, schedule, c)
                if schedule == api.SCHEDULE_PER_BLOCK:
                    mine = [(b["cost"], b["op"], b["all_before"], b["stored_before"], b["to_check"]) for b in res.blocks]
                    assert mine == [p for p in ref.progress if p[1] != "A"]
