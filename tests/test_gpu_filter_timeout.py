"""The filter's put-off look-back, made to run out: with two to four polls allowed and
one range per CTA (no next range to put the look-back off behind) the walk meets
ranges that have not published yet.  ghb_sync reports it, and the context then gives
the oracle's result."""
import numpy as np
import pytest

from ghive_b200 import abi
from ghive_b200._lib import GhbError
from oracle import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("polls", [2, 4])
def test_put_off_lookback_runs_out(polls):
    import torch

    from ghive_b200.ops import Context
    d = np.random.default_rng(polls).integers(0, 2526, 3_000_000, dtype=np.int32)
    pred = abi.Pred.leaf(abi.FILTER_LT, 0, a=1263)
    dd = torch.from_numpy(d).cuda()
    with Context(0) as ctx:
        ctx.set_spin_limit(polls)
        codes = []
        for _ in range(8):
            try:
                ctx.filter(pred, [dd])
            except GhbError as e:
                codes.append(e.code)
        assert codes and set(codes) == {abi.ERR_TIMEOUT}
        ctx.set_spin_limit(0)
        outs, k = ctx.filter(pred, [dd])
        sel = oracle.filter_rows(pred, [d])
        assert k == len(sel) and np.array_equal(outs[0][0].cpu().numpy(), d[sel])
