"""The general write pass of the join probe: every join type over duplicated
and unique, dense and spread keys, more payloads than a slot holds, NULL maps
and sentinels, and an output that is too short.  Pairs equal the oracle's."""
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


@pytest.mark.parametrize("jt", [abi.INNER_JOIN, abi.LEFT_OUTER_JOIN, abi.LEFT_SEMI_JOIN])
@pytest.mark.parametrize("dup", [1, 2, 40])
@pytest.mark.parametrize("spread", [False, True])
@pytest.mark.parametrize("n", [1, 127, 128, 1025, 70_001])
def test_pairs_and_payloads(ctx, jt, dup, spread, n):
    g = np.random.default_rng(n + dup)
    nb = 600
    key = np.arange(nb, dtype=np.int64) * (1_000_003 if spread else 1)
    bkey = g.permutation(np.concatenate([key, np.repeat(key[:7], dup - 1)]))
    fk = np.where(g.random(n) < 0.3, -5, key[g.integers(0, 60, n)])
    pnull = g.random(n) < 0.1
    m = len(bkey)
    bp = [g.integers(0, 1 << 40, m, dtype=np.int64), g.random(m), g.integers(0, 99, m, dtype=np.int32), g.random(m)]
    bnull = g.random(m) < 0.2
    pp = [g.integers(0, 99, n, dtype=np.int32), g.random(n)]
    pr, br = oracle.hash_join(bkey, (fk, pnull), jt)
    t = ctx.join_build(dev(bkey), build_payload=[dev(bp[0]), dev(bp[1]), dev(bp[2]), (dev(bp[3]), dev(bnull))])
    r = ctx.join_probe(t, (dev(fk), dev(pnull)), jt, probe_payload=[dev(pp[0]), (dev(pp[1]), dev(pnull))],
                       capacity=max(1, len(pr)))
    assert r["rows"] == len(pr)
    gp, gb = r["probe_rowid"].cpu().numpy(), r["build_rowid"].cpu().numpy()
    assert np.all(np.diff(gp) >= 0)
    o1, o2 = np.lexsort((gb, gp)), np.lexsort((br, pr))
    assert np.array_equal(gp[o1], pr[o2]) and np.array_equal(gb[o1], br[o2])
    hit = gb >= 0
    for j, x in enumerate(bp):
        v, nul = [c.cpu().numpy() for c in r["build"][j]]
        exp_null = ~hit | (bnull[gb] if j == 3 else False)
        assert np.array_equal(nul, exp_null)
        assert np.array_equal(v[~exp_null].view(np.uint8), x[gb[~exp_null]].view(np.uint8))
    for j, x in enumerate(pp):
        v, nul = [c.cpu().numpy() for c in r["probe"][j]]
        exp_null = pnull[gp] if j == 1 else np.zeros(len(gp), bool)
        assert np.array_equal(nul, exp_null)
        assert np.array_equal(v[~exp_null].view(np.uint8), x[gp[~exp_null]].view(np.uint8))
    t.free()


def test_short_output_is_reported(ctx):
    from ghive_b200._lib import GhbError
    t = ctx.join_build(dev(np.repeat(np.arange(50, dtype=np.int64), 3)))
    with pytest.raises(GhbError) as e:
        ctx.join_probe(t, dev(np.arange(50, dtype=np.int64)), capacity=149)
    assert e.value.code == abi.ERR_CAPACITY
    assert ctx.join_probe(t, dev(np.arange(50, dtype=np.int64)), capacity=150)["rows"] == 150
    t.free()
