"""The engine's limits hold on the small levels too: the rows and cache bytes of the configuration, and the
size of the hash set.  A search that passes one of them has one answer, whether one CTA ran its small levels
or the level kernel did, alone or in a call of any number of instances."""
import numpy as np
import pytest

import oracle as O
from ltlb200 import api, gen
from helpers import on_the_fly_cases

pytestmark = pytest.mark.gpu


def key(r):
    return r.status, r.cost, r.all_ltls, r.rows, r.on_the_fly


@pytest.mark.parametrize("limit,workers,count,max_cost", [("rows", 4, 300, 14), ("bytes", 2000, 2000, 3)])
def test_batch_calls_of_any_size_keep_the_cache_limits(limit, workers, count, max_cost):
    """Caches that hold exactly the rows up to a level: the next one overflows, nothing of it is stored, and
    the search goes on as one engine's does.  (Two instances a multiprocessor give the small-level CTAs levels
    of a few thousand candidates, enough to reach the find; more slots than CTAs give a CTA more than a slot's
    cache; 3 instances go to the slots at once.)"""
    inst = gen.generate(24, 2, 20, 20, 8, 16, 0.5, 7)
    _, cases = on_the_fly_cases(inst, (1,) * 8)
    assert len(cases) == 3
    for k, cap in cases:
        kw = dict(slots_log2=12, max_traces=512)
        kw.update(dict(cache_bytes=256 << 20, max_rows=cap) if limit == "rows" else dict(cache_bytes=cap * 40 * 8))
        with api.Engine(**kw) as e:
            want = e.learn(inst, neg_type=1, max_cost=max_cost)
        if k < max_cost:
            assert want.on_the_fly and want.rows == cap
        with api.Batch(workers=workers, **kw) as b:
            for n in (3, count):
                for r in b.learn([inst] * n, neg_type=1, max_cost=max_cost):
                    assert key(r) == key(want), (k, n)


# one proposition or two, costs under which many levels are small: 1,095 rows up to cost 19 with at most 200
# operand pairs in a level; 1,170 up to cost 10 with levels of up to a few thousand candidates
FULL = [(2, (2, 2, 11, 11, 2, 2, 2, 11), 19, 1), (1, (1, 1, 4, 4, 1, 1, 1, 4), 10, 300)]


@pytest.mark.parametrize("props,costs,max_cost,count", FULL)
def test_full_hash_set_on_small_levels(props, costs, max_cost, count):
    rng = np.random.default_rng(7)
    lens, bits, _, _ = gen._draw(rng, 24, props, 8, 30, 0.5)
    letters = "".join(sorted(gen.DEFAULT_LETTERS[:props]))
    steps, offs = gen._pack(letters, list(lens), list(bits))
    inst = gen.Instance(12, 12, letters, steps, offs)
    opts = dict(costs=costs, max_cost=max_cost, stop_at_found=False, neg_type=1)
    ref = O.learn(inst, cache_rows=1 << 14, **opts)
    assert 1024 < ref.num_rows < 2048
    kw = dict(cache_bytes=64 << 20, max_rows=1 << 15, max_traces=64)
    for log2, status in ((10, api.TABLE_FULL), (11, None)):
        with api.Engine(slots_log2=log2, **kw) as e:
            levels = e.learn(inst, schedule=api.SCHEDULE_PER_BLOCK, **opts)
            assert status is None or levels.status == status
            assert e.learn(inst, **opts).status == levels.status
        with api.Batch(workers=4, slots_log2=log2, **kw) as b:
            for r in b.learn([inst] * count, **opts):
                assert r.status == levels.status
                assert status is not None or r.rows == ref.num_rows
