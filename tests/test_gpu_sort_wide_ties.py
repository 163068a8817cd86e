"""ORDER BY keys wider than 64 bits whose rows agree in the leading 64 and
differ below them, at every number of leading digits that the sort may choose:
with many (ASCII digits, a far outlier) few bits are left to the finish.

The permutation is compared with the oracle's stable one, row for row."""
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


@pytest.mark.parametrize("digits,n", [(9, 1_000_000), (10, 20_000), (10, 1_000_000), (11, 1_000_000),
                                      (12, 1_000_000), (10, 4_000_000)])
@pytest.mark.parametrize("order", [abi.ASC, abi.DESC])
def test_decimal_strings(ctx, digits, n, order):
    """Numbers of 9 to 12 digits as STRING keys: two 8-byte parts."""
    g = np.random.default_rng(digits * 10 + order)
    v = g.integers(0, 10 ** digits, n)
    chars = np.empty((n, digits), np.uint8)
    rest = v.copy()
    for i in reversed(range(digits)):
        chars[:, i] = ord("0") + rest % 10
        rest //= 10
    start = np.arange(n, dtype=np.int32) * digits
    s = ("string", chars.reshape(-1), np.stack([start, start + digits], 1).reshape(-1))
    perm = oracle.sort_perm([s], [order], threads=8)
    _, _, rid = ctx.sort([("string", dev(s[1]), dev(s[2]))], [order], rowid=True)
    assert np.array_equal(rid.cpu().numpy(), perm)


# of 62 bits (one far outlier) the values use `width`: the first 62 - width
# say nothing, and eight bits more than the rows' need one more leading digit
@pytest.mark.parametrize("width", [23, 31, 39, 47])
@pytest.mark.parametrize("n", [9000, 100_000])
@pytest.mark.parametrize("orders", [[abi.ASC, abi.ASC], [abi.DESC, abi.ASC]])
def test_outlier_then_a_second_key(ctx, width, n, orders):
    """A BIGINT with one far outlier and each value about twice, then an INT or a
    nullable BIGINT that alone orders the repeats."""
    g = np.random.default_rng(width)
    a = g.choice(g.integers(0, 1 << width, n // 2), n)
    a[n // 3] = (1 << 62) - 1
    pay = np.arange(n, dtype=np.int32)
    b = g.integers(-2 ** 31, 2 ** 31 - 1, n, dtype=np.int32)
    perm = oracle.sort_perm([a, b], orders, threads=8)
    ok, op, _ = ctx.sort([dev(a), dev(b)], orders, payload=[dev(pay)])
    assert np.array_equal(op[0][0].cpu().numpy(), perm)
    assert np.array_equal(ok[0][0].cpu().numpy(), a[perm]) and np.array_equal(ok[1][0].cpu().numpy(), b[perm])
    c, null = g.integers(0, 1 << 40, n), g.random(n) < 0.2
    perm = oracle.sort_perm([a, (c, null)], orders, threads=8)
    _, op, _ = ctx.sort([dev(a), (dev(c), dev(null))], orders, payload=[dev(pay)])
    assert np.array_equal(op[0][0].cpu().numpy(), perm)
