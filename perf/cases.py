"""The framework's measured calls: what a user's program asks of it, over the sizes it is used at.

A case is a dict of plain values.  `prepare` makes what such a program has in hand before the
call (seeded traces on the host, a warm engine or batch handle on the GPU), `run` is one pass
through the public Python API, and `work` says what one pass cannot do without.

Kinds
  learn     one learn on a warm engine: to the minimal formula, or (stop False) every level up
            to max_cost in full, as the uniqueness comparison and the label collection do
  sequence  many small learns one after another on one engine, as divide-and-conquer does
  batch     many instances through the batch call
  evaluate  one formula on every trace, as the divide-and-conquer driver checks sub-formulas
  train     the block-order scorer's training on collected records

Traces are Bernoulli bits labelled by a hidden random formula (drawn until no single letter
separates them), or near misses (negatives are positives with one to three flipped bits).
Outputs are the values that do not depend on the order in which warps reach the hash set:
status, cost, the reference's candidate count, per-level counts.  The formula's text is one of
several of equal cost and is not among them.
"""
import math

import numpy as np
import torch

from __graft_entry__ import load_package

load_package()
from ltlb200 import api, gen, learned  # noqa: E402

UNIT = (1,) * 8
SCALE_COSTS = (1, 1, 1, 1, 1, 2, 2, 3)  # letter, ~, &, |, X, F, G, U: the scale workload's

# Distinct characteristic sets of cost 1, 2, ... over so many propositions, on enough long random
# traces to tell all formulas of these costs apart (unit costs, every formula may be negated).
UNIQUES = {
    1: (1, 4, 9, 17, 56, 172, 450, 1297, 3962, 12072),
    2: (2, 8, 21, 77, 333, 1200, 4712, 19837),
    3: (3, 12, 37, 181, 876, 3867, 19399, 97900),
    4: (4, 16, 57, 329, 1729, 8954, 52000),
    5: (5, 20, 81, 521, 2936, 17247),
}
SCALE_UNIQUES = (5, 10, 45, 177, 696, 3102, 13133, 59095, 263943)  # five propositions, SCALE_COSTS


def _learn(name, props, npos, nneg, lmin, lmax, *, fsize=8, max_cost=8, stop=True, neg_type=1, key="exact",
           schedule="fused", order="plain", costs="unit", p_bit=0.5, depth=0):
    return dict(name=name, kind="learn", props=props, npos=npos, nneg=nneg, lmin=lmin, lmax=lmax, fsize=fsize,
                max_cost=max_cost, stop=stop, neg_type=neg_type, key=key, schedule=schedule, order=order, costs=costs,
                p_bit=p_bit, depth=depth)


def listed():
    return [
        # the smallest real call: one learn of a few dozen short traces, launches and latency only
        _learn("one_small", 2, 20, 20, 8, 16, fsize=7, depth=4),
        # the reference's own regime (few short traces, its uniqueness keys, letters negated only)
        _learn("reference_keys", 3, 10, 2, 5, 8, max_cost=6, stop=False, neg_type=2, key="ref"),
        # the reference's progress lines: one launch per (operator, split) block
        _learn("per_block", 3, 8, 8, 7, 7, max_cost=6, stop=False, schedule="per_block"),
        # divide and conquer: the sub-problems of a run, one after another on one engine
        dict(name="subproblems", kind="sequence", count=24, props_max=3, traces_max=32, lmin=5, lmax=24, fsize_max=7,
             max_cost=7, depth=4),
        # a thousand traces, every level to cost 8 (about 120 thousand rows of 8 KB)
        _learn("thousand_census", 3, 500, 500, 16, 32, fsize=9, max_cost=8, stop=False),
        # the same shape batched, each instance to its minimal formula
        dict(name="thousand_batch", kind="batch", count=16, slots=8, props_min=3, props_max=3, traces_min=500,
             traces_max=500, lmin=16, lmax=32, fsize_min=9, fsize_max=9, max_cost=8, key="exact", cache_mb=1536,
             slots_log2=20, depth=6),
        # many small and ragged instances in one call
        dict(name="many_small", kind="batch", count=512, slots=48, props_min=2, props_max=4, traces_min=8,
             traces_max=256, lmin=4, lmax=40, fsize_min=3, fsize_max=8, max_cost=7, key="exact", cache_mb=384,
             slots_log2=18, depth=4),
        # the largest rows: 4000 long traces, uneven costs, exact uniqueness
        _learn("scale_exact", 5, 2000, 2000, 32, 63, fsize=12, max_cost=9, stop=False, costs="scale", p_bit=0.3),
        # odd sizes with 64-bit-fingerprint uniqueness
        _learn("odd_hash64", 4, 1501, 1497, 12, 40, fsize=10, max_cost=7, stop=False, key="hash64", p_bit=0.2),
        # the learned block order on near misses (no separating formula within the bound)
        _learn("learned_order", 4, 1000, 1000, 20, 48, max_cost=7, stop=False, order="learned", p_bit=0.3),
        # a formula checked on a large corpus
        dict(name="evaluate_corpus", kind="evaluate", props=3, npos=50000, nneg=50000, lmin=10, lmax=10, fsize=20),
        # the scorer's training
        dict(name="train_scorer", kind="train", records=16384, epochs=2, batch=1024),
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi + 0.49)))))))


def _max_cost_for(props, n, budget_bytes):
    c = 3
    while c < len(UNIQUES[props]) and sum(UNIQUES[props][:c + 1]) * n * 8 <= budget_bytes and c < 8:
        c += 1
    return c


def draw(rng):
    kind = rng.choice(["learn", "learn", "census", "census", "sequence", "batch", "evaluate", "train"])
    if kind in ("learn", "census"):
        props = rng.randint(1, 5)
        npos, nneg = _log_int(rng, 4, 2000), _log_int(rng, 4, 2000)
        lmin = rng.randint(4, 32)
        lmax = rng.randint(max(lmin, 8), 63)
        key = rng.choice(["exact", "exact", "hash64"])
        if kind == "learn":
            c = _learn("", props, npos, nneg, lmin, lmax, fsize=rng.randint(5, 9), key=key, depth=5,
                       max_cost=_max_cost_for(props, npos + nneg, 1 << 30), neg_type=rng.choice([1, 2]))
        else:
            c = _learn("", props, npos, nneg, lmin, lmax, max_cost=_max_cost_for(props, npos + nneg, 1 << 30),
                       stop=False, key=key, neg_type=rng.choice([1, 2]))
    elif kind == "sequence":
        c = dict(kind="sequence", count=rng.randint(4, 24), props_max=rng.randint(2, 3),
                 traces_max=_log_int(rng, 6, 64), lmin=rng.randint(4, 8), lmax=rng.randint(9, 40),
                 fsize_max=rng.randint(5, 7), max_cost=7, depth=4)
    elif kind == "batch":
        tmin = _log_int(rng, 4, 64)
        tmax = _log_int(rng, tmin + 4, 500)
        pmin = rng.randint(1, 3)
        c = dict(kind="batch", count=_log_int(rng, 6, 512 if tmax <= 256 else 24), slots=rng.choice([8, 16, 48]),
                 props_min=pmin, props_max=rng.randint(pmin, 3 if tmax > 256 else 4), traces_min=tmin, traces_max=tmax,
                 lmin=rng.randint(4, 10), lmax=rng.randint(11, 48), fsize_min=3, fsize_max=rng.randint(5, 9),
                 max_cost=7, key=rng.choice(["exact", "exact", "hash64"]), cache_mb=384, slots_log2=18, depth=4)
    elif kind == "evaluate":
        lmin = rng.randint(1, 12)
        c = dict(kind="evaluate", props=rng.randint(1, 6), npos=_log_int(rng, 5, 50000), nneg=_log_int(rng, 5, 40000),
                 lmin=lmin, lmax=lmin, fsize=rng.randint(2, 24))
    else:
        c = dict(kind="train", records=_log_int(rng, 500, 16000), epochs=rng.randint(1, 2),
                 batch=rng.choice([256, 1000, 1024]))
    c.pop("name", None)
    return c


# ---------------------------------------------------------------- inputs
def _pack(letters, lens, bits):
    """The instance arrays of traces given as [n, lmax, props] bits and their lengths."""
    offsets = np.zeros(len(lens) + 1, dtype=np.int32)
    offsets[1:] = np.cumsum(lens)
    shifts = np.array([ord(c) - 97 for c in letters], dtype=np.uint32)
    masks = (bits.astype(np.uint32) << shifts[None, None, :]).sum(axis=2, dtype=np.uint32)
    live = np.arange(bits.shape[1])[None, :] < np.asarray(lens)[:, None]
    return masks[live], offsets


def _draw_traces(rng, m, props, lmin, lmax, p_bit):
    lens = rng.integers(lmin, lmax + 1, size=m)
    bits = rng.random((m, lmax, props), dtype=np.float32) < p_bit
    bits &= (np.arange(lmax)[None, :] < lens[:, None])[:, :, None]
    weights = np.uint64(1) << np.arange(lmax, dtype=np.uint64)
    atoms = np.stack([(bits[:, :, j] * weights).sum(axis=1, dtype=np.uint64) for j in range(props)])
    mask = (np.uint64(1) << lens.astype(np.uint64)) - np.uint64(1)
    return lens, bits, atoms, mask


def _letters(props):
    return "".join(sorted(gen.DEFAULT_LETTERS[:props]))


def _instance(rng, props, npos, nneg, lmin, lmax, fsize, p_bit=0.5):
    """Traces labelled by a hidden random formula; redrawn while one letter separates them."""
    for attempt in range(400):
        if attempt % 40 == 0:
            lens, bits, atoms, mask = _draw_traces(rng, 4 * (npos + nneg) + 64, props, lmin, lmax, p_bit)
        f = gen.random_formula(rng, fsize, props)
        lab = (gen.eval_cs(f, atoms, mask) & np.uint64(1)).astype(bool)
        pos, neg = np.nonzero(lab)[0][:npos], np.nonzero(~lab)[0][:nneg]
        if len(pos) < npos or len(neg) < nneg:
            continue
        if attempt < 360:
            first = (atoms & np.uint64(1)).astype(bool)
            if any(first[j][pos].all() and not first[j][neg].any() for j in range(props)):
                continue
        at = np.concatenate([pos, neg])
        steps, offsets = _pack(_letters(props), lens[at], bits[at])
        return gen.Instance(npos, nneg, _letters(props), steps, offsets, gen.formula_str(f, _letters(props)))
    raise RuntimeError("no hidden formula fills the quotas")


def _engine_for(case, n, max_rows):
    log2 = 16
    while (1 << log2) < 3 * max_rows:
        log2 += 1
    pitch = max(4, (n + 3) // 4 * 4)
    return api.Engine(slots_log2=log2, cache_bytes=(max_rows + 1024) * pitch * 8, max_rows=max_rows + 1024,
                      max_traces=max(n, 1))


def _rows(case):
    per = SCALE_UNIQUES if case["costs"] == "scale" else UNIQUES[case["props"]]
    return per[:case["max_cost"]]


def _options(case):
    return dict(costs=SCALE_COSTS if case.get("costs") == "scale" else UNIT, max_cost=case["max_cost"],
                neg_type=case.get("neg_type", 1), stop_at_found=case.get("stop", True),
                key_mode={"exact": api.KEY_EXACT, "ref": api.KEY_REF, "hash64": api.KEY_HASH64}[case.get("key", "exact")],
                schedule=api.SCHEDULE_PER_BLOCK if case.get("schedule") == "per_block" else api.SCHEDULE_FUSED,
                order=api.ORDER_LEARNED if case.get("order") == "learned" else api.ORDER_PLAIN)


def prepare(case, seed):
    rng = np.random.default_rng(seed)
    kind = case["kind"]
    if kind == "learn":
        n = case["npos"] + case["nneg"]
        if case["order"] == "learned":
            inst = gen.generate_near_miss(seed, case["props"], case["npos"], case["nneg"], case["lmin"], case["lmax"],
                                          case["p_bit"])
        else:
            inst = _instance(rng, case["props"], case["npos"], case["nneg"], case["lmin"], case["lmax"], case["fsize"],
                             case["p_bit"])
        eng = _engine_for(case, n, int(1.25 * sum(_rows(case))))
        if case["order"] == "learned":
            eng.set_scorer(learned.load_scorer())
        return dict(kind=kind, engine=eng, inst=inst, opts=_options(case), stop=case["stop"])
    if kind == "sequence":
        insts = [_instance(rng, int(rng.integers(2, case["props_max"] + 1)),
                           int(rng.integers(3, case["traces_max"] + 1)), int(rng.integers(3, case["traces_max"] + 1)),
                           case["lmin"], case["lmax"], int(rng.integers(4, case["fsize_max"] + 1)))
                 for _ in range(case["count"])]
        eng = api.Engine(slots_log2=20, cache_bytes=256 << 20, max_rows=1 << 18, max_traces=2 * case["traces_max"])
        return dict(kind=kind, engine=eng, insts=insts, opts=_options(case))
    if kind == "batch":
        insts = [_instance(rng, int(rng.integers(case["props_min"], case["props_max"] + 1)),
                           int(rng.integers(case["traces_min"], case["traces_max"] + 1)),
                           int(rng.integers(case["traces_min"], case["traces_max"] + 1)), case["lmin"], case["lmax"],
                           int(rng.integers(case["fsize_min"], case["fsize_max"] + 1)))
                 for _ in range(case["count"])]
        handle = api.Batch(workers=case["slots"], slots_log2=case["slots_log2"], cache_bytes=case["cache_mb"] << 20,
                           max_rows=1 << 20, max_traces=2 * case["traces_max"])
        return dict(kind=kind, batch=handle, insts=insts, opts=_options(case))
    if kind == "evaluate":
        n = case["npos"] + case["nneg"]
        lens, bits, _, _ = _draw_traces(rng, n, case["props"], case["lmin"], case["lmax"], 0.5)
        steps, offsets = _pack(_letters(case["props"]), lens, bits)
        inst = gen.Instance(case["npos"], case["nneg"], _letters(case["props"]), steps, offsets)
        f = gen.formula_str(gen.random_formula(rng, case["fsize"], case["props"]), _letters(case["props"]))
        return dict(kind=kind, inst=inst, formula=f)
    x, y = _records(case, seed)
    return dict(kind=kind, params=learned.init_params(seed), x=x, y=y, epochs=case["epochs"], batch=case["batch"],
                seed=seed)


def _records(case, seed):
    """Feature vectors in the ranges the planner makes (one-hot operator, ratios, log sizes) and labels
    that a noisy rule on them gives, about one in ten positive."""
    rng = np.random.default_rng(seed)
    count = case["records"]
    x = rng.random((count, api.SCORER_FEATURES), dtype=np.float32)
    x[:, :7] = np.eye(7, dtype=np.float32)[rng.integers(0, 7, size=count)]
    x[:, 27:31] = rng.random((count, 4)) < 0.4
    x[:, 31] = 1.0
    z = 3.0 * x[:, 17] * x[:, 20] + x[:, 6] - x[:, 13] + 0.3 * rng.standard_normal(count)
    return x, (z > np.quantile(z, 0.9)).astype(np.float32)


# ---------------------------------------------------------------- one pass
def _census(r):
    return {"head": np.array([r.status, r.cost, r.all_ltls, r.rows], dtype=np.int64),
            "levels": np.array([[v["cost"], v["candidates"], v["uniques"]] for v in r.levels], dtype=np.int64),
            "blocks": np.array([[b["cost"], api.OPS.index(b["op"]), b["left_cost"], b["right_cost"],
                                 b["stored_before"], b["all_before"], b["to_check"]] for b in r.blocks],
                               dtype=np.int64)}


def run(state):
    kind = state["kind"]
    if kind == "learn":
        r = state["engine"].learn(state["inst"], **state["opts"])
        return _census(r) if not state["stop"] else np.array([r.status, r.cost, r.all_ltls], dtype=np.int64)
    if kind == "sequence":
        rs = [state["engine"].learn(i, **state["opts"]) for i in state["insts"]]
        return np.array([[r.status, r.cost, r.all_ltls] for r in rs], dtype=np.int64)
    if kind == "batch":
        rs = state["batch"].learn(state["insts"], **state["opts"])
        return np.array([[r.status, r.cost, r.all_ltls] for r in rs], dtype=np.int64)
    if kind == "evaluate":
        cs, holds = api.evaluate(state["inst"], state["formula"])
        return {"cs": cs.view(np.int64), "holds": holds}
    params, curve = api.scorer_train(state["params"], state["x"], state["y"], epochs=state["epochs"],
                                     batch=state["batch"], pos_weight=9.0, seed=state["seed"])
    return {"params": params, "loss": curve}


# ---------------------------------------------------------------- what a pass cannot do without
def work(case):
    kind = case["kind"]
    if kind in ("learn", "sequence", "batch"):
        # every distinct CS is written once (row, parents, hash slot) and, below the last level, read
        # once as an operand; searches that stop at a find are counted to their typical depth
        if kind == "learn":
            n, count = case["npos"] + case["nneg"], 1
            per = _rows(case)
        else:
            n = case["traces_max"] if kind == "sequence" else (case["traces_min"] + case["traces_max"])
            count = case["count"]
            per = UNIQUES[case["props_max"]]
        if case["depth"]:
            per = per[:case["depth"]]
        row = 8 * n
        return {"bytes": count * (sum(per) * (row + 16) + sum(per[:-1]) * row), "flops": 0}
    if kind == "evaluate":
        n = case["npos"] + case["nneg"]
        return {"bytes": n * (4 * (case["lmin"] + case["lmax"]) // 2 + 4 + 8 + 1), "flops": 0}
    return {"bytes": case["epochs"] * case["records"] * 4 * (api.SCORER_FEATURES + 1),
            "flops": case["epochs"] * case["records"] * 6.0 * (32 * 64 + 64 * 64 + 64)}


# ---------------------------------------------------------------- 64-bit values of the computed numbers
def exact(case, seed):
    """The scorer's training in 64 bits (the other kinds return whole numbers)."""
    if case["kind"] != "train":
        return None
    x, y = _records(case, seed)
    x, y = x.astype(np.float64), y.astype(np.float64)
    p = learned.init_params(seed).astype(np.float64)
    nf, h = 32, 64
    cuts = np.cumsum([0, h * nf, h, h * h, h, h, 1])
    is_weight = np.zeros(p.size, dtype=bool)
    for q in (0, 2, 4):
        is_weight[cuts[q]:cuts[q + 1]] = True
    m, v = np.zeros_like(p), np.zeros_like(p)
    perm, s, step, curve = list(range(len(y))), seed & (2 ** 64 - 1), 0, []

    def rand():  # splitmix64, the shuffle's generator
        nonlocal s
        s = (s + 0x9E3779B97F4A7C15) & (2 ** 64 - 1)
        z = s
        z = ((z ^ (z >> 30)) * 0xBF58476D1CE4E5B9) & (2 ** 64 - 1)
        z = ((z ^ (z >> 27)) * 0x94D049BB133111EB) & (2 ** 64 - 1)
        return z ^ (z >> 31)

    for _ in range(case["epochs"]):
        for i in range(len(y) - 1, 0, -1):
            j = rand() % (i + 1)
            perm[i], perm[j] = perm[j], perm[i]
        total = 0.0
        for first in range(0, len(y), case["batch"]):
            at = perm[first:first + case["batch"]]
            a, t = x[at], y[at]
            w1, b1, w2, b2, w3, b3 = (p[cuts[q]:cuts[q + 1]] for q in range(6))
            w1, w2 = w1.reshape(h, nf), w2.reshape(h, h)
            h1 = np.maximum(a @ w1.T + b1, 0)
            h2 = np.maximum(h1 @ w2.T + b2, 0)
            z = h2 @ w3 + b3
            w = np.where(t > 0.5, 9.0, 1.0)
            total += float((w * (np.maximum(z, 0) - z * t + np.log1p(np.exp(-np.abs(z))))).sum())
            dz = w * (1 / (1 + np.exp(-z)) - t) / len(at)
            d2 = np.where(h2 > 0, dz[:, None] * w3, 0)
            d1 = np.where(h1 > 0, d2 @ w2, 0)
            g = np.concatenate([(d1.T @ a).ravel(), d1.sum(0), (d2.T @ h1).ravel(), d2.sum(0), dz @ h2, [dz.sum()]])
            step += 1
            m = 0.9 * m + 0.1 * g
            v = 0.999 * v + 0.001 * g * g
            p = p - 2e-3 * (m / (1 - 0.9 ** step)) / (np.sqrt(v / (1 - 0.999 ** step)) + 1e-8)
        curve.append(total / len(y))
    return {"params": torch.from_numpy(p), "loss": torch.tensor(curve, dtype=torch.float64)}
