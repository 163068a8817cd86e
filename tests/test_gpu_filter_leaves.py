"""Filter leaves as interval tests, in every mode, at the edges of the column
types and of the literals; trees of several leaves; sizes around a tile and a
claimed range.  Rows and order equal the oracle's."""
import numpy as np
import pytest

from ghive_b200 import abi
from oracle import oracle

pytestmark = pytest.mark.gpu

MODES = [abi.FILTER_EQ, abi.FILTER_LE, abi.FILTER_GE, abi.FILTER_LT, abi.FILTER_GT, abi.FILTER_RANGE,
         abi.FILTER_EQ_RANGE, abi.FILTER_NOT_EQ, abi.FILTER_NOT_RANGE, abi.FILTER_NOT_EQ_RANGE, abi.FILTER_NOT_NULL]
I32, I64 = np.iinfo(np.int32), np.iinfo(np.int64)


@pytest.fixture(scope="module")
def ctx():
    from ghive_b200.ops import Context
    c = Context(0)
    yield c
    c.close()


def dev(a):
    import torch
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


def check(ctx, pred, cols, nulls=(None, None, None)):
    sel = oracle.filter_rows(pred, [c if m is None else (c, m) for c, m in zip(cols, nulls)])
    outs, k = ctx.filter(pred, [dev(c) if m is None else (dev(c), dev(m)) for c, m in zip(cols, nulls)])
    assert k == len(sel)
    for c, m, (v, isnull) in zip(cols, nulls, outs):
        assert np.array_equal(v.cpu().numpy().view(np.uint8), c[sel].view(np.uint8))
        assert np.array_equal(isnull.cpu().numpy(), np.zeros(len(sel), bool) if m is None else m[sel])


@pytest.mark.parametrize("mode", MODES)
def test_every_mode_at_the_edges(ctx, mode):
    g = np.random.default_rng(mode)
    n = 4097
    i = g.choice(np.array([I32.min, I32.min + 1, -1, 0, 7, 8, I32.max - 1, I32.max], dtype=np.int32), n)
    j = g.choice(np.array([I64.min, I64.min + 1, I32.min - 1, -1, 0, 7, I32.max + 1, I64.max - 1, I64.max]), n)
    x = g.choice(np.array([-np.inf, -1e300, -0.0, 0.0, 7.0, 7.5, 1e300, np.inf, np.nan]), n)
    m = g.random(n) < 0.2
    for a, b in [(7, 8), (0, 0), (8, 7), (I64.min, I64.max), (I64.max, I64.min), (I32.max, I32.max + 1),
                 (I32.min - 5, I32.min), (I64.max, I64.max), (I64.min, I64.min)]:
        for col in range(2):
            check(ctx, abi.Pred.leaf(mode, col, a=a, b=b), [i, j, x], (m, None, None))
            check(ctx, abi.Pred.leaf(mode, col, a=a, b=b), [i, j, x], (None, m, m))
    for a, b in [(0.0, 7.25), (-0.5, 7.0), (np.inf, -np.inf)]:
        for col in range(3):
            check(ctx, abi.Pred.leaf(mode, col, a=float(a), b=float(b)), [i, j, x], (m, m, m))


@pytest.mark.parametrize("n", [1, 31, 255, 2047, 2048, 2049, 8191, 8192, 8193, 3 * 8192 + 77, 9_000_001])
def test_trees_at_tile_and_range_edges(ctx, n):
    g = np.random.default_rng(n)
    i = g.integers(0, 1000, n, dtype=np.int32)
    j = g.integers(-50, 50, n, dtype=np.int64)
    x = g.normal(0, 1, n)
    m = g.random(n) < 0.1
    leaf = abi.Pred.leaf
    one = abi.Pred.and_(leaf(abi.FILTER_EQ_RANGE, 0, a=100, b=700), leaf(abi.FILTER_LT, 1, a=20))
    two = abi.Pred.or_(abi.Pred.and_(one, leaf(abi.FILTER_GT, 2, a=0.25)),
                       abi.Pred.and_(leaf(abi.FILTER_NOT_NULL, 1), leaf(abi.FILTER_GE, 0, a=0, col2=1)))
    check(ctx, one, [i, j, x], (None, m, None))
    check(ctx, two, [i, j, x], (m, m, None))
    check(ctx, None, [i, j, x], (None, None, m))
