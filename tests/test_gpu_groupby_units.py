"""GROUP BY results at the sizes where the finalize changes its unit (tables
of 2^17 slots and more), and key packing at row counts and addresses where its
16-byte loads do not apply.  Groups equal the oracle's."""
import numpy as np
import pytest

from ghive_b200 import abi
from oracle import oracle

pytestmark = pytest.mark.gpu
REL_TOL = 1e-12   # DOUBLE sums against the oracle's sequential sum, as in test_gpu_ops


@pytest.fixture(scope="module")
def ctx():
    from ghive_b200.ops import Context
    c = Context(0)
    yield c
    c.close()


def dev(a):
    import torch
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


def check(ctx, cols, nulls, keys, aggs, max_groups, shift=0):
    """Compares every group; with `shift` the device columns start that many
    rows into their buffers."""
    def up(a):
        return dev(np.concatenate([a[:shift], a]))[shift:] if shift else dev(a)
    hcols = [c if m is None else (c, m) for c, m in zip(cols, nulls)]
    ok, oa = oracle.filter_groupby(None, hcols, keys, aggs)
    gk, ga, g = ctx.filter_groupby(None, [up(c) if m is None else (up(c), up(m.astype(np.uint8))) for c, m in
                                          zip(cols, nulls)], keys, aggs, capacity=max_groups, max_groups=max_groups)
    assert g == len(ok[0][0])

    def order(kcols):
        return np.lexsort([x for v, n in reversed(kcols) for x in (np.where(n, 0, v), n)])
    gk = [(v.cpu().numpy(), n.cpu().numpy()) for v, n in gk]
    ok = [(v, np.zeros(len(v), bool) if n is None else n.astype(bool)) for v, n in ok]
    a, b = order(gk), order(ok)
    for (v, n), (w, m) in zip(gk, ok):
        assert np.array_equal(n[a], m[b]) and np.array_equal(v[a][~n[a]], w[b][~m[b]])
    for (v, n), (w, m) in zip(ga, oa):
        v, n = v.cpu().numpy()[a], n.cpu().numpy()[a]
        m = np.zeros(len(w), bool) if m is None else m.astype(bool)
        assert np.array_equal(n, m[b])
        v, w = v[~n], w[b][~m[b]]
        if v.dtype == np.float64:
            assert np.all(np.abs(v - w) <= REL_TOL * np.abs(w))
        else:
            assert np.array_equal(v, w)


@pytest.mark.parametrize("groups", [1, 255, 40_000, 65_536, 65_537, 150_000])
def test_every_aggregate_around_the_unit_change(ctx, groups):
    g = np.random.default_rng(groups)
    n = 400_000
    key = g.integers(0, groups, n, dtype=np.int64) * 7919 - 5
    q, x, d = g.integers(-99, 99, n, dtype=np.int64), np.round(g.uniform(1, 1e5, n), 2), g.integers(0, 999, n, dtype=np.int32)
    m = g.random(n) < 0.5
    aggs = [(abi.CNT, -1), (abi.CNT, 2), (abi.SUM, 1), (abi.SUM, 2), (abi.AVG, 2), (abi.MIN, 2), (abi.MAX, 3), (abi.MIN, 1)]
    check(ctx, [key, q, x, d], [None, None, m, None], [0], aggs, groups)
    check(ctx, [key, q], [g.random(n) < 0.1, None], [0], [(abi.SUM, 1)], groups + 1)   # a NULL group; an odd record


# Around the number of groups from which the fold leaves more of an SM to its
# L1 and halves its shared table for that (LONG keys 2048 slots, INT 4096).
@pytest.mark.parametrize("dtype", [np.int32, np.int64])
@pytest.mark.parametrize("groups", [4096, 4097, 8192, 8193, 16_385, 32_768, 32_769])
def test_shared_memory_left_to_the_cache(ctx, groups, dtype):
    rng = np.random.default_rng(groups)
    n = 3 * groups + 17
    k = rng.permutation(np.arange(n) % groups).astype(dtype) - 5
    qty, price, d = (rng.integers(1, 51, n), rng.integers(100, 10_000, n) / 100.0,
                     rng.integers(0, 2526, n, dtype=np.int32))
    aggs = [(abi.CNT, -1), (abi.SUM, 1), (abi.SUM, 2), (abi.AVG, 2), (abi.MIN, 3), (abi.MAX, 3)]
    check(ctx, [k, qty, price, d], [None] * 4, [0], aggs, groups)


@pytest.mark.parametrize("n", [1, 3, 4, 5, 1023, 70_001])
@pytest.mark.parametrize("shift", [0, 1])
def test_packed_keys_off_the_vector_path(ctx, n, shift):
    g = np.random.default_rng(n)
    a = g.integers(-4, 4, n, dtype=np.int32)
    b = g.integers(1 << 40, (1 << 40) + 9, n, dtype=np.int64)
    x = g.choice(np.array([0.5, 0.75, 3.0]), n)
    v = g.integers(0, 50, n, dtype=np.int64)
    m1, m2 = g.random(n) < 0.2, g.random(n) < 0.2
    for keys, nulls in [([0, 1], (m1, m2, None, None)), ([2, 0], (None, None, m1, None)), ([1, 0, 2], (m2, None, None, None))]:
        check(ctx, [a, b, x, v], nulls, keys, [(abi.CNT, -1), (abi.SUM, 3)], 9 * 10 * 4, shift if n > shift else 0)
