"""A sort whose look-back gives up while the error of an earlier call is still on
the context: the sort stops by a word of its own, not by the status word, which
keeps the earlier error.  (Reading on, it would take row indices that no pass wrote.)"""
import numpy as np
import pytest

from ghive_b200 import abi
from ghive_b200._lib import GhbError
from oracle import oracle

pytestmark = pytest.mark.gpu


def dev(a):
    import torch
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


# a key of one word with its payload carried, one sorted by every digit and gathered,
# and one wider than a word
@pytest.mark.parametrize("form", ["carried", "skewed", "wide"])
def test_an_earlier_error_does_not_hide_it(form):
    from ghive_b200.ops import Context
    g = np.random.default_rng(5)
    n = 4_000_000
    k = g.integers(0, 1 << 62, n)
    if form == "skewed":
        k[: n // 2] = 77
    keys = [k, g.integers(-2 ** 31, 2 ** 31 - 1, n, dtype=np.int32)] if form == "wide" else [k]
    pay = [g.integers(0, 9, n)] * (1 if form == "carried" else 2)
    dk, dp = [dev(x) for x in keys], [dev(x) for x in pay]
    with Context(0) as ctx:
        ctx.set_spin_limit(1)
        for _ in range(4):
            ctx.filter(None, [dk[0]], capacity=1, sync=False)   # leaves GHB_ERR_CAPACITY
            with pytest.raises(GhbError) as e:
                ctx.sort(dk, payload=dp)
            assert e.value.code in (abi.ERR_CAPACITY, abi.ERR_TIMEOUT)
        ctx.set_spin_limit(0)
        ok, op, _ = ctx.sort(dk, payload=dp)
        perm = oracle.sort_perm(keys, threads=8)
        for (got, _), x in zip(ok + op, keys + pay):
            assert np.array_equal(got.cpu().numpy(), x[perm])
