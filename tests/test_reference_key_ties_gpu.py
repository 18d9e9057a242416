"""Which formula a CS keeps under the reference's keys: of a level's candidates with one CS, a row's parents are
those of a candidate in the first of the blocks that hold one, in the reference's order (~, & by split, | by split,
X, F, G, U by split).  Up to 126 positions in all the keys hold whole CSs; 127 positions are the first size of the
relaxed keys.  Small levels, the level kernel, rows of 512 words and more, wide rows, both schedules.  The oracle
stores candidates in the reference's order one at a time."""
import numpy as np
import pytest

import oracle as O
from ltlb200 import api, gen

pytestmark = pytest.mark.gpu

UNIT = (1,) * 8


def instance(seed, lens, props):
    rng = np.random.default_rng(seed)
    letters = "".join(sorted(gen.DEFAULT_LETTERS[:props]))
    steps = np.zeros(sum(lens), dtype=np.uint32)
    for c in letters:
        steps |= (rng.random(len(steps)) < 0.5).astype(np.uint32) << np.uint32(ord(c) - 97)
    offs = np.concatenate([[0], np.cumsum(lens)]).astype(np.int32)
    return gen.Instance(len(lens) - len(lens) // 2, len(lens) // 2, letters, steps, offs)


def lengths(total, n, nonempty):
    out = [total // nonempty] * nonempty
    out[0] += total - sum(out)
    return out + [0] * (n - nonempty)


@pytest.mark.parametrize("schedule", [api.SCHEDULE_FUSED, api.SCHEDULE_PER_BLOCK])
@pytest.mark.parametrize("total,n,nonempty,props,max_cost,costs,neg", [
    (78, 12, 12, 3, 6, UNIT, 2), (78, 12, 12, 3, 5, UNIT, 1), (126, 14, 14, 2, 7, UNIT, 1),
    (126, 40, 40, 3, 7, (1, 1, 1, 1, 1, 2, 2, 3), 1), (100, 10, 10, 3, 8, (1, 2, 2, 1, 3, 1, 2, 2), 1), (126, 520, 20, 2, 6, UNIT, 1),
    (126, 1100, 18, 2, 5, UNIT, 1), (126, 2200, 18, 2, 5, UNIT, 1)])
def test_first_block_keeps_the_row(total, n, nonempty, props, max_cost, costs, neg, schedule):
    inst = instance(total + n, lengths(total, n, nonempty), props)
    assert int(inst.lengths.sum()) == total
    ref = O.learn(inst, costs=costs, max_cost=max_cost, neg_type=neg, key_mode=O.KEY_REF3, stop_at_found=False,
                  cache_rows=1 << 17)
    cost_of = lambda starts, r: int(np.searchsorted(starts, r, side="right")) - 1

    def blocks(rows, ops, left, right, starts):
        out = {}
        for r in range(len(inst.alphabet), len(rows)):
            op = int(ops[r])
            ends = [cost_of(starts, int(left[r]))] + ([cost_of(starts, int(right[r]))] if op in (1, 2, 6) else [])
            out[rows[r].tobytes()] = (cost_of(starts, r), op, min(ends))
        return out

    want = blocks(ref.rows, ref.row_op, ref.row_left, ref.row_right, np.array(ref.level_start[:max_cost + 2]))
    with api.Engine(slots_log2=18, cache_bytes=1 << 30, max_rows=1 << 16, max_traces=max(n, 64)) as e:
        for rlx in (1, 3):
            for _ in range(3):
                res = e.learn(inst, costs=costs, max_cost=max_cost, neg_type=neg, key_mode=api.KEY_REF, rlx_type=rlx,
                              stop_at_found=False, schedule=schedule)
                assert (res.device_flags, res.all_ltls, res.rows) == (0, ref.all_ltls, ref.num_rows)
                starts = np.array(e.level_starts(max_cost + 2))
                rows, par = e.read_rows(0, int(starts[max_cost + 1]))
                mine = blocks(rows, (par >> np.uint64(60)) & np.uint64(7), (par >> np.uint64(30)) & np.uint64(0x3FFFFFFF),
                              par & np.uint64(0x3FFFFFFF), starts[:max_cost + 2])
                differ = [(want.get(k), b) for k, b in mine.items() if want.get(k) != b]
                assert not differ, (rlx, len(differ), len(mine), differ[:5])


@pytest.mark.parametrize("rlx", [1, 2, 3])
@pytest.mark.parametrize("total", [126, 127])
def test_sizes_at_the_edge_of_the_keys(total, rlx):
    """The progress lines (a shared key stays with the first block that has it) and the counts up to cost 4."""
    inst = instance(total, lengths(total, 14, 14), 3)
    ref = O.learn(inst, max_cost=4, neg_type=1, key_mode=rlx, stop_at_found=False)
    opts = dict(max_cost=4, neg_type=1, key_mode=api.KEY_REF, rlx_type=rlx, stop_at_found=False)
    with api.Engine(slots_log2=18, cache_bytes=64 << 20, max_rows=1 << 16) as e:
        res = e.learn(inst, schedule=api.SCHEDULE_PER_BLOCK, **opts)
        assert [(b["cost"], b["op"], b["all_before"], b["stored_before"], b["to_check"]) for b in res.blocks] == \
            [p for p in ref.progress if p[1] != "A"]
        full = e.learn(inst, **opts)
        assert (full.status, full.all_ltls, full.rows) == (res.status, res.all_ltls, res.rows)
