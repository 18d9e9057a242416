"""The device time a batch reports for an instance is all of it: the pass of one CTA over its small levels, and the
slot's from set-up to the result, whichever of them the call used."""
import numpy as np
import pytest

from ltlb200 import api, gen

pytestmark = pytest.mark.gpu


def test_small_level_pass_counts():
    """One slot, so that nothing runs beside an instance there.  Three instances go to the slot at once; 80 have
    their pass first, which does not reach cost 5, and then go to the slot.  A pass that ends at cost 2 is shorter
    than theirs and is reported alone."""
    inst = gen.generate(11, 3, 450, 450, 16, 60, 0.5, 9)
    kw = dict(neg_type=1, stop_at_found=False)
    ms = lambda res: float(np.median([r.device_ms for r in res]))
    with api.Batch(workers=1, slots_log2=16, cache_bytes=1 << 30, max_rows=1 << 15, max_traces=1024) as b:
        b.learn([inst] * 80, max_cost=5, **kw)
        alone, both, local = [], [], []
        for _ in range(3):
            alone.append(ms(b.learn([inst] * 3, max_cost=5, **kw)))
            both.append(ms(b.learn([inst] * 80, max_cost=5, **kw)))
            local.append(ms(b.learn([inst] * 80, max_cost=2, **kw)))
    alone, both, local = (float(np.median(x)) for x in (alone, both, local))
    assert both >= alone + 0.5 * local, (alone, both, local)
