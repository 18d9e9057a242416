"""The engine's limits hold on the small levels too: the rows and cache bytes of the configuration.  A
search that passes one of them has one answer, whether one CTA ran its small levels
or the level kernel did, alone or in a call of any number of instances."""
import pytest

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
