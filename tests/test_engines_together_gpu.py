"""Engines of several threads on one GPU at the same time.

Each learn is a set-up launch and one launch of the level kernel, whose blocks start whenever an SM is
free: beside another engine's kernel some start late, when their own search is about to end or has ended.
Every learn's result is the one its engine gives alone."""
import threading

import pytest

import oracle as O
from ltlb200 import api, gen

pytestmark = pytest.mark.gpu


def test_engines_on_threads_learn_as_alone():
    insts = [gen.generate(300 + s, 3, 30, 30, 6, 20, 0.5, 7) for s in range(6)]
    insts += [gen.generate(500 + s, 3, 120, 120, 8, 30, 0.5, 7) for s in range(3)]
    kw = dict(slots_log2=20, cache_bytes=256 << 20, max_rows=1 << 18)
    with api.Engine(**kw) as e:
        want = [e.learn(i, neg_type=1, max_cost=8) for i in insts]
    got, errors = {}, []

    def work(k):
        try:
            with api.Engine(**kw) as e:
                for rep in range(8):
                    for j in range(len(insts)):
                        q = (j + k) % len(insts)
                        r = e.learn(insts[q], neg_type=1, max_cost=8)
                        got.setdefault((k, q), []).append(r)
        except Exception as x:  # handed to the main thread
            errors.append(x)

    threads = [threading.Thread(target=work, args=(k,)) for k in range(3)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors
    for (k, q), rs in got.items():
        for r in rs:
            assert (r.status, r.cost, r.all_ltls, r.device_flags) == (want[q].status, want[q].cost, want[q].all_ltls, 0)
            if r.status == api.FOUND:
                assert O.separates(r.formula, insts[q]) and O.formula_cost(r.formula) == r.cost
