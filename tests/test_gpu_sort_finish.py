"""Sorts whose radix passes cover the leading digits only: the finish orders
each run of equal leading digits, whole tiles and long runs among them.

Every result is compared with the oracle's stable permutation, bit for bit.
"""
import numpy as np
import pytest

from ghive_b200 import abi
from oracle import oracle

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    from ghive_b200.ops import Context
    c = Context(0)
    yield c
    c.close()


def dev(a):
    import torch
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


def check(ctx, keys, orders=None, payload=(), nulls=None):
    perm = oracle.sort_perm([k if nulls is None or nulls[i] is None else (k, nulls[i]) for i, k in enumerate(keys)],
                            orders, threads=8)
    dk = [dev(k) if nulls is None or nulls[i] is None else (dev(k), dev(nulls[i])) for i, k in enumerate(keys)]
    ok, op, rid = ctx.sort(dk, orders, payload=[dev(x) for x in payload], rowid=len(payload) != 1)
    if rid is not None:
        assert np.array_equal(rid.cpu().numpy(), perm)
    for i, k in enumerate(keys):
        got, isnull = ok[i][0].cpu().numpy(), ok[i][1].cpu().numpy()
        exp_null = np.zeros(len(k), bool) if nulls is None or nulls[i] is None else nulls[i][perm]
        assert np.array_equal(isnull, exp_null)
        assert np.array_equal(got[~exp_null].view(np.uint8), k[perm][~exp_null].view(np.uint8))
    for x, (v, _) in zip(payload, op):
        assert np.array_equal(v.cpu().numpy().view(np.uint8), x[perm].view(np.uint8))


@pytest.mark.parametrize("n", [9000, 10 * 2048 - 1, 10 * 2048, 10 * 2048 + 1, 64 * 4096, 300_001])
@pytest.mark.parametrize("bits", [20, 41, 62])
def test_random_keys_at_tile_edges(ctx, n, bits):
    g = np.random.default_rng(n + bits)
    k = g.integers(0, 1 << bits, n, dtype=np.int64)
    check(ctx, [k], payload=[np.arange(n, dtype=np.int32)])                 # 32-bit value carried
    check(ctx, [k], [abi.DESC], payload=[g.random(n)])                      # 64-bit value carried
    check(ctx, [k], payload=[g.random(n), np.arange(n, dtype=np.int32)])    # row index carried, columns gathered


@pytest.mark.parametrize("run", [40, 1000, 2048, 3200, 5000, 60_000])
@pytest.mark.parametrize("order", ["random", "same", "two"])
def test_a_few_long_runs_among_even_keys(ctx, run, order):
    """Runs of equal leading digits too few for the sample to weigh: longer
    than the test for order, than a tile, than a tile and the rows read past it."""
    g = np.random.default_rng(run)
    n = 3_000_000
    k = g.integers(0, 1 << 46, n, dtype=np.int64)
    for i in range(3):
        low = {"random": g.integers(0, 1 << 14, run), "same": np.full(run, 77), "two": g.integers(0, 2, run)}[order]
        k[g.choice(n, run, replace=False)] = ((g.integers(0, 1 << 20) << 26) | low)
    check(ctx, [k], payload=[np.arange(n, dtype=np.int32)])


def test_keys_whose_leading_digits_say_little(ctx):
    """A second key that follows the first (a date and its timestamp), one
    far outlier, few distinct values, and a nullable double in between."""
    g = np.random.default_rng(5)
    n = 500_000
    day = g.integers(0, 300, n, dtype=np.int32)
    stamp = day.astype(np.int64) * 86_400_000 + g.integers(0, 86_400_000, n)
    check(ctx, [day, stamp], payload=[np.arange(n, dtype=np.int32)])
    far = g.integers(0, 1 << 20, n, dtype=np.int64)
    far[n // 2] = 1 << 60
    check(ctx, [far], [abi.DESC], payload=[np.arange(n, dtype=np.int32)])
    few = g.choice(np.array([1, 5, 1 << 40, (1 << 40) + 3]), n)
    check(ctx, [day, few])
    x = np.round(g.normal(0, 1e4, n), 2)
    xn = g.random(n) < 0.1
    check(ctx, [x, day], [abi.DESC, abi.ASC], nulls=[xn, None], payload=[stamp, far])


def test_sorted_and_reversed_input(ctx):
    n = 200_000
    k = np.arange(n, dtype=np.int64) * 1_000_003
    check(ctx, [k], payload=[np.arange(n, dtype=np.int32)])
    check(ctx, [k[::-1].copy()], payload=[np.arange(n, dtype=np.int32)])


@pytest.mark.parametrize("ties", ["none", "below", "equal"])
@pytest.mark.parametrize("orders", [[abi.ASC, abi.ASC], [abi.DESC, abi.ASC]])
def test_keys_wider_than_a_word(ctx, ties, orders):
    """Keys of 69 and 128 bits: sorted by the leading 64 when those tell the
    rows apart, by every bit when rows differ only below them or are equal."""
    g = np.random.default_rng(11)
    n = 300_007
    i = g.integers(0, 24, n, dtype=np.int32)
    j = g.integers(np.iinfo(np.int64).min, np.iinfo(np.int64).max, n, dtype=np.int64)
    if ties != "none":
        a, b = g.choice(n, (2, 400), replace=False)
        i[b], j[b] = i[a], j[a] ^ (1 if ties == "below" else 0)
    pay = [np.arange(n, dtype=np.int32), g.random(n)]
    check(ctx, [i, j], orders, payload=pay)
    check(ctx, [j, g.integers(np.iinfo(np.int64).min, np.iinfo(np.int64).max, n, dtype=np.int64)], orders,
          payload=pay[:1])
    check(ctx, [j, i], orders, payload=pay, nulls=[g.random(n) < 0.001, g.random(n) < 0.1])
