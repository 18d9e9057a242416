"""The kernels that sizes choose, at the edges of their ranges, against the CPU oracle.

The small levels' CTA takes rows of at most 1024 words and levels that fit its tables; wide rows (tiles of
two rows, then of one) begin where three 4-row tiles no longer fit the shared memory.  Integer work:
comparisons are exact."""
import numpy as np
import pytest

import oracle as O
from ltlb200 import api, gen
from helpers import row_set

pytestmark = pytest.mark.gpu


def traces(seed, n, lmin=1, lmax=63, props=2):
    rng = np.random.default_rng(seed)
    lens, bits, _, _ = gen._draw(rng, n, props, lmin, lmax, 0.5)
    letters = "".join(sorted(gen.DEFAULT_LETTERS[:props]))
    steps, offs = gen._pack(letters, list(lens), list(bits))
    return gen.Instance(n - n // 2, n // 2, letters, steps, offs)


def check(eng, inst, max_cost, costs=(1,) * 8, neg_type=1, key=api.KEY_EXACT):
    res = eng.learn(inst, costs=costs, max_cost=max_cost, stop_at_found=False, neg_type=neg_type, key_mode=key)
    ref = O.learn(inst, costs=costs, max_cost=max_cost, stop_at_found=False, neg_type=neg_type, cache_rows=1 << 17)
    assert res.device_flags == 0 and res.all_ltls == ref.all_ltls
    starts = eng.level_starts(max_cost + 2)
    rows, par = eng.read_rows(0, starts[max_cost + 1])
    mask = (np.uint64(1) << inst.lengths.astype(np.uint64)) - np.uint64(1)
    for c in range(costs[0], max_cost + 1):
        assert row_set(rows[starts[c]:starts[c + 1]]) == row_set(ref.level_rows(c)), c
    for r in range(len(inst.alphabet), len(rows)):
        p = int(par[r])
        op, a, b = (p >> 60) & 7, (p >> 30) & 0x3FFFFFFF, p & 0x3FFFFFFF
        assert np.array_equal(O.apply_op(op, rows[a], rows[b] if op in (1, 2, 6) else None, mask)[0], rows[r])


@pytest.mark.parametrize("key", [api.KEY_EXACT, api.KEY_HASH64])
@pytest.mark.parametrize("n", [2, 16, 17, 64, 65, 128, 1021, 1024, 1025])
def test_small_level_sizes(n, key):
    with api.Engine(slots_log2=18, cache_bytes=512 << 20, max_rows=1 << 17) as eng:
        check(eng, traces(n, n), 7 if n < 100 else 5, key=key)


@pytest.mark.parametrize("costs,neg", [((1, 1, 1, 1, 1, 2, 2, 3), 1), ((1, 2, 2, 1, 3, 1, 2, 2), 2), ((2, 1, 3, 2, 1, 1, 2, 3), 1)])
def test_small_level_costs(costs, neg):
    with api.Engine(slots_log2=18, cache_bytes=256 << 20, max_rows=1 << 17) as eng:
        check(eng, traces(5, 30, props=3), 8, costs=costs, neg_type=neg)


def test_duplicate_letters_and_letter_spans():
    """A letter that never differs from another stays a row; letters far apart take wider step masks."""
    rng = np.random.default_rng(8)
    for letters in ("ab", "aj", "az"):
        steps, offs = [], [0]
        for _ in range(20):
            ln = int(rng.integers(1, 12))
            b = rng.random(ln) < 0.5
            steps += [(1 << (ord(letters[0]) - 97)) * int(x) | (1 << (ord(letters[1]) - 97)) * int(x) for x in b]
            offs.append(offs[-1] + ln)
        inst = gen.Instance(10, 10, letters, np.array(steps, dtype=np.uint32), np.array(offs, dtype=np.int32))
        with api.Engine(slots_log2=16, cache_bytes=64 << 20, max_rows=1 << 15) as eng:
            check(eng, inst, 5)


@pytest.mark.parametrize("n", [2132, 2140, 6600, 8300, 12800])
def test_wide_rows(n):
    with api.Engine(slots_log2=16, cache_bytes=1 << 30, max_rows=1 << 14, max_traces=n) as eng:
        check(eng, traces(n, n, props=2), 4)


def test_batch_takes_small_and_large_instances():
    """Results of a batch are a single engine's, whichever kernel ended each instance's search."""
    insts = [gen.generate(s, 2 + s % 3, 6 + 5 * (s % 7), 9 + 3 * (s % 11), 4, 30, 0.5, 3 + s % 6) for s in range(120)]
    insts += [traces(900 + k, n) for k, n in enumerate((2, 300, 1025))]
    for key in (api.KEY_EXACT, api.KEY_HASH64):
        opts = dict(max_cost=6, neg_type=1, key_mode=key)
        with api.Batch(workers=5, slots_log2=18, cache_bytes=256 << 20, max_rows=1 << 16) as b, \
                api.Engine(slots_log2=18, cache_bytes=256 << 20, max_rows=1 << 16) as eng:
            got = b.learn(insts, **opts)
            for inst, r in zip(insts, got):
                w = eng.learn(inst, **opts)
                assert (r.status, r.cost, r.all_ltls) == (w.status, w.cost, w.all_ltls)
                if r.status == api.FOUND:
                    assert O.separates(r.formula, inst) and O.formula_cost(r.formula) == r.cost
                else:
                    assert (r.rows, r.evaluated) == (w.rows, w.evaluated)


@pytest.mark.parametrize("depth", [1, 31, 32, 33, 150])
def test_evaluate_depth(depth):
    """Formulas whose evaluation stack stays in shared memory and ones whose stack does not."""
    inst = traces(depth, 131, lmin=1, props=2)
    f = inst.alphabet[0]
    for k in range(depth - 1):
        f = f"({inst.alphabet[k % 2]}){'&|U'[k % 3]}({f})" if k % 5 else f"(X({inst.alphabet[1]}))U({f})"
    cs, holds = api.evaluate(inst, f)
    atoms = inst.atom_cs()
    mask = (np.uint64(1) << inst.lengths.astype(np.uint64)) - np.uint64(1)
    v = atoms[0]
    for k in range(depth - 1):
        a = atoms[k % 2]
        v = ((a & v, a | v, gen._until(a, v))[k % 3]) if k % 5 else gen._until(atoms[1] >> np.uint64(1), v)
    assert np.array_equal(cs, v & mask) and np.array_equal(holds, (v & np.uint64(1)).astype(bool))


@pytest.mark.parametrize("count", [1, 15, 16, 17, 4735, 4737, 9600])
def test_scorer_gradient_sizes(count):
    """Groups of 16 records, the last ragged, and more groups than CTAs (296): the oracle's gradient,
    within the bounds the scorer's other tests use (BF16 operands; relative L2 1e-2, loss 1e-4)."""
    import scorer_oracle as S
    rng = np.random.default_rng(count)
    x = rng.random((count, api.SCORER_FEATURES), dtype=np.float32)
    y = (rng.random(count) < 0.3).astype(np.float32)
    p = (rng.standard_normal(api.SCORER_PARAMS) * 0.2).astype(np.float32)
    g, loss = api.scorer_grad(p, x, y, pos_weight=2.0)
    wg, wl = S.grad(p, x, y, 2.0)
    assert np.linalg.norm(g - wg) <= 1e-2 * np.linalg.norm(wg) and abs(loss - wl) <= 1e-4 * max(1.0, abs(wl))
