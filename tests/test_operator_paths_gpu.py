"""The operators as every path of the enumerator applies them, on one word: the level kernel's units, its sweeps over
wide rows, the small levels, and the formula evaluator's in natural order.  The device compares them with one another
(bit 63 of a result is set where two differ) and the oracle's result is exact.  Words of every length from an empty
trace to 63 steps: all ones, all zeros, single positions, alternating and random ones."""
import numpy as np
import pytest

import oracle as O
from ltlb200 import api

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("op", range(7))
def test_paths_agree_at_every_length(op):
    lens = np.arange(64)
    mask = np.array([(1 << int(k)) - 1 for k in lens], dtype=np.uint64)
    rng = np.random.default_rng(op)
    last = np.array([1 << max(int(k) - 1, 0) for k in lens], dtype=np.uint64)
    words = [np.zeros(64, np.uint64), mask, last, np.ones(64, np.uint64), np.full(64, 0x5555555555555555, np.uint64),
             np.full(64, 0x2AAAAAAAAAAAAAAA, np.uint64), ~last, ~np.ones(64, np.uint64)]
    words += [rng.integers(0, 2 ** 63, size=64, dtype=np.uint64) for _ in range(8)]
    words += [words[-1] & words[-2] & words[-3], words[-1] | words[-2] | words[-3]]
    words = np.stack(words) & mask
    a = np.repeat(words, len(words), axis=0)
    b = np.tile(words, (len(words), 1))
    out, out2, fp = api.device_apply_op(op, a, b if op in (1, 2, 6) else None, mask)
    for r in range(len(a)):
        o1, o2 = O.apply_op(op, a[r], b[r] if op in (1, 2, 6) else None, mask)
        assert np.array_equal(out[r], o1), (op, r)
        assert int(fp[r]) == O.fp64(o1)
        if op == 6:
            assert np.array_equal(out2[r], o2) and int(fp[len(a) + r]) == O.fp64(o2)
