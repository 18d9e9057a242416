"""What a search leaves out once its level has a find: the operators whose blocks come after it, also where one
entry runs several operators on a pair (equal costs), in the level kernel and on the small levels."""
import pytest

import oracle as O
from ltlb200 import api, gen

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("left_tile", [2, 4, 8])
@pytest.mark.parametrize("seed,cost", [(34, 7), (8, 9)])
def test_fused_entries_stop_at_a_find(seed, cost, left_tile):
    """A unary operator finds, in a block between | and U, and unary entries are first in the queue: the U blocks,
    a quarter of the level and more, are left out but for the items then in work."""
    inst = gen.generate(seed, 3, 500, 500, 16, 32, 0.5, 9)
    with api.Engine(slots_log2=22, cache_bytes=6 << 30, max_rows=1 << 20, left_tile=left_tile) as e:
        found = e.learn(inst, neg_type=1)
        full = e.learn(inst, neg_type=1, max_cost=cost, stop_at_found=False)
    assert found.status == api.FOUND and found.cost == cost and found.found_op in (3, 4, 5)
    assert O.separates(found.formula, inst) and O.formula_cost(found.formula) == cost
    assert found.evaluated < 0.85 * full.evaluated


@pytest.mark.parametrize("seed", [17, 24, 32])
def test_small_levels_stop_at_a_find(seed):
    """300 instances give a CTA levels of a few thousand candidates, several rounds each."""
    inst = gen.generate(seed, 2, 20, 20, 8, 16, 0.5, 7)
    ref = O.learn(inst, neg_type=1)
    kw = dict(neg_type=1, max_cost=ref.cost)
    with api.Batch(workers=4, slots_log2=14, cache_bytes=256 << 20, max_rows=1 << 14, max_traces=64) as b:
        found = b.learn([inst] * 300, **kw)
        full = b.learn([inst] * 300, stop_at_found=False, **kw)
    for r, f in zip(found, full):
        assert r.status == api.FOUND and (r.cost, r.all_ltls) == (ref.cost, ref.all_ltls)
        assert O.separates(r.formula, inst) and O.formula_cost(r.formula) == r.cost
        assert r.evaluated < f.evaluated
