"""Runs of equal leading digits of every length that the sort's finish treats
in its own way (a thread, a warp, the CTA, the list of long runs), in a tile and
over its end, and what one of them may cost."""
import time

import numpy as np
import pytest

from ghive_b200 import abi
from oracle import oracle

pytestmark = pytest.mark.gpu

RUNS = [16, 17, 31, 32, 33, 64, 65, 127, 128, 129, 255, 256, 257, 1000, 1023, 1024, 1025, 2047, 2048, 2500]


@pytest.fixture(scope="module")
def ctx():
    from ghive_b200.ops import Context
    c = Context(0)
    yield c
    c.close()


def dev(a):
    import torch
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


def with_runs(g, n, runs, low):
    """n keys of 46 bits in [2^45, 2^46) but for runs below them, in key order
    from the first row on, that differ in their `low` lowest bits only."""
    k = g.integers(1 << 45, 1 << 46, n, dtype=np.int64)
    at, first = g.permutation(n), 0
    for i, run in enumerate(runs):
        k[at[first:first + run]] = (i << 26) + g.integers(0, 1 << low, run)
        first += run
    return k


@pytest.mark.parametrize("low", [0, 3, 14])
@pytest.mark.parametrize("shift", [0, 1900])
def test_runs_of_every_length(ctx, low, shift):
    """Each length alone at the front of a sort (`shift` rows of other runs before
    it: the run then crosses a tile's end), and all of them one after another."""
    g = np.random.default_rng(low + shift)
    n = 1_000_000
    for runs in [[1] * shift + [r] for r in RUNS] + [[1] * shift + RUNS]:
        k = with_runs(g, n, runs, low)
        perm = oracle.sort_perm([k], threads=8)
        _, op, _ = ctx.sort([dev(k)], payload=[dev(np.arange(n, dtype=np.int32))])
        assert np.array_equal(op[0][0].cpu().numpy(), perm), runs[shift:]


@pytest.mark.parametrize("orders", [[abi.ASC, abi.ASC], [abi.ASC, abi.DESC]])
@pytest.mark.parametrize("distinct", [1, 3, 1 << 20])
def test_runs_of_a_wide_key(ctx, orders, distinct):
    """Rows that agree in the leading 64 bits (or in all but three of them) and are
    told apart by a second key."""
    g = np.random.default_rng(distinct)
    n = 1_000_000
    for run in [17, 32, 33, 128, 129, 1024, 1025, 2000]:
        a = g.integers(1 << 61, 1 << 62, n, dtype=np.int64)
        a[g.permutation(n)[:run]] = g.integers(0, distinct, run) & 3
        b = g.integers(-2 ** 31, 2 ** 31 - 1, n, dtype=np.int32)
        perm = oracle.sort_perm([a, b], orders, threads=8)
        _, _, rid = ctx.sort([dev(a), dev(b)], orders, rowid=True)
        assert np.array_equal(rid.cpu().numpy(), perm), run


def best_ms(fn):
    import torch
    best = 1e9
    for i in range(8):
        torch.cuda.synchronize()
        t = time.perf_counter()
        fn()
        torch.cuda.synchronize()
        best = min(best, (time.perf_counter() - t) * 1e3)
    return best


@pytest.mark.parametrize("run", [500, 1000, 2000, 2500])
def test_one_run_does_not_hold_a_sort_up(ctx, run):
    """A sort of a million rows takes about 0.18 ms; every row of one unordered run
    against every other by one warp would add 0.1 ms at 500 rows, 1.7 ms at 2000.
    Half as much again as without the run is allowed."""
    g = np.random.default_rng(run)
    n = 1_000_000
    pay = dev(np.arange(n, dtype=np.int32))
    plain, with_run = (dev(with_runs(g, n, r, 14)) for r in ([], [run]))
    t0 = best_ms(lambda: ctx.sort([plain], payload=[pay], with_nulls=False))
    t1 = best_ms(lambda: ctx.sort([with_run], payload=[pay], with_nulls=False))
    assert t1 < 1.5 * t0, (t0, t1)


def test_one_run_of_a_wide_key_does_not_hold_a_sort_up(ctx):
    """The same with 500 rows that agree in the leading 64 bits of a wide key: about
    0.23 ms without them.  Two and a half times that is allowed (a sort by every bit
    takes twice); a comparison by the columns of every row with every other took 6 ms."""
    g = np.random.default_rng(3)
    n = 1_000_000
    a = g.integers(1 << 61, 1 << 62, n, dtype=np.int64)
    b = dev(g.integers(-2 ** 31, 2 ** 31 - 1, n, dtype=np.int32))
    plain = dev(a)
    a[g.permutation(n)[:500]] = 5
    with_run = dev(a)
    t0 = best_ms(lambda: ctx.sort([plain, b], rowid=True))
    t1 = best_ms(lambda: ctx.sort([with_run, b], rowid=True))
    assert t1 < 2.5 * t0, (t0, t1)
