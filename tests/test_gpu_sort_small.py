"""ORDER BY of a few thousand rows (one CTA): every row count class and its
edges, keys of one and of two 64-bit words, NULLs, all types.  Equal to the
oracle's stable permutation, bit for bit."""
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


@pytest.mark.parametrize("n", [1, 2, 31, 33, 511, 512, 513, 1024, 1025, 4096, 4097, 8191, 8192, 8193])
def test_sizes_types_and_nulls(ctx, n):
    g = np.random.default_rng(n)
    i = g.integers(-5, 300, n, dtype=np.int32)
    j = g.integers(np.iinfo(np.int64).min, np.iinfo(np.int64).max, n, dtype=np.int64)   # 64 bits alone
    x = np.round(g.normal(0, 100, n), 1)
    m, mj = g.random(n) < 0.2, g.random(n) < 0.1
    pay = [g.integers(0, 9, n, dtype=np.int64), g.random(n), np.arange(n, dtype=np.int32)]
    A, D = abi.ASC, abi.DESC
    F, L, N = abi.NULLS_FIRST, abi.NULLS_LAST, abi.NULLS_DEFAULT
    for keys, nulls, orders, no, npay in [
            ([i], [None], [A], [N], 1), ([i, x], [m, None], [D, A], [N, N], 3), ([j], [None], [D], [N], 0),
            ([i, j], [m, mj], [A, D], [L, F], 2), ([j, x, i], [mj, m, None], [A, A, D], [F, L, N], 3),
            ([np.full(n, 7)], [None], [A], [N], 1), ([np.full(n, 7), i % 3], [np.ones(n, bool), None], [A, D], [N, N], 1)]:
        keys = [k.astype(np.int32) if k.dtype == np.int32 else k for k in keys]
        perm = oracle.sort_perm([k if z is None else (k, z) for k, z in zip(keys, nulls)], orders, no)
        ok, op, rid = ctx.sort([dev(k) if z is None else (dev(k), dev(z)) for k, z in zip(keys, nulls)], orders, no,
                               payload=[dev(p) for p in pay[:npay]], rowid=True)
        assert np.array_equal(rid.cpu().numpy(), perm)
        for k, z, (v, isnull) in zip(keys, nulls, ok):
            exp = np.zeros(n, bool) if z is None else z[perm]
            assert np.array_equal(isnull.cpu().numpy(), exp)
            assert np.array_equal(v.cpu().numpy()[~exp].view(np.uint8), k[perm][~exp].view(np.uint8))
        for p, (v, _) in zip(pay, op):
            assert np.array_equal(v.cpu().numpy().view(np.uint8), p[perm].view(np.uint8))


def test_sentinel_nulls(ctx):
    from ghive_b200.ops import Sentinel
    g = np.random.default_rng(3)
    k = g.choice(np.array([1, 2, np.iinfo(np.int64).max, -4]), 700)
    ok, _, rid = ctx.sort([Sentinel(dev(k))], [abi.DESC], rowid=True)
    null = k == np.iinfo(np.int64).max
    perm = oracle.sort_perm([(k, null)], [abi.DESC])
    assert np.array_equal(rid.cpu().numpy(), perm)
    assert np.array_equal(ok[0][0].cpu().numpy(), k[perm])
    assert np.array_equal(ok[0][1].cpu().numpy(), null[perm])


@pytest.mark.parametrize("run", [2, 47, 48, 49, 200])
def test_runs_of_equal_leading_digits(ctx, run):
    """64-bit keys of which `run` share their leading 16 bits: around the
    longest run whose order is counted, and beyond."""
    g = np.random.default_rng(run)
    n = 5000
    k = g.integers(np.iinfo(np.int64).min, np.iinfo(np.int64).max, n, dtype=np.int64)
    k[g.choice(n, run, replace=False)] = (5 << 48) + g.integers(0, 9, run)
    pay = np.arange(n, dtype=np.int32)
    ok, op, _ = ctx.sort([dev(k)], payload=[dev(pay)])
    perm = oracle.sort_perm([k])
    assert np.array_equal(ok[0][0].cpu().numpy(), k[perm]) and np.array_equal(op[0][0].cpu().numpy(), pay[perm])
