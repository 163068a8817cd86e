"""Join keys with many build rows met by few probe rows: a warp walks such chains
together, the others a row a round.  Pairs and payloads equal the oracle's."""
import time

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


# further rows of a chain around the 16 that are walked together and the 32 of a
# step; chains of a warp (128 probe rows) around the four that are
@pytest.mark.parametrize("dup", [16, 17, 18, 32, 33, 34, 65, 1000])
@pytest.mark.parametrize("hot", [1, 3, 4, 5, 9])
@pytest.mark.parametrize("jt", [abi.INNER_JOIN, abi.LEFT_OUTER_JOIN])
def test_few_long_chains(ctx, dup, hot, jt):
    g = np.random.default_rng(dup * 10 + hot)
    n, nb = 1000, 3000
    bkey = g.permutation(np.concatenate([np.arange(nb), np.repeat([5, 6, 7], [dup - 1, dup // 2, 1])])) * 1_000_003
    fk = g.integers(10, nb + 300, n) * 1_000_003
    for first in (0, 128, 512, 640):   # warps with `hot` rows of chains of three lengths
        fk[first + g.choice(128, hot, replace=False)] = g.choice([5, 5, 6, 7], hot) * 1_000_003
    m = len(bkey)
    bp = [g.integers(0, 1 << 40, m), g.random(m), g.integers(0, 99, m, dtype=np.int32), g.random(m)]
    bnull = g.random(m) < 0.2
    pp = g.integers(0, 99, n, dtype=np.int32)
    pr, br = oracle.hash_join(bkey, fk, jt)
    t = ctx.join_build(dev(bkey), build_payload=[dev(bp[0]), dev(bp[1]), dev(bp[2]), (dev(bp[3]), dev(bnull))])
    r = ctx.join_probe(t, dev(fk), jt, probe_payload=[dev(pp)], capacity=len(pr))
    gp, gb = r["probe_rowid"].cpu().numpy(), r["build_rowid"].cpu().numpy()
    assert r["rows"] == len(pr) and np.all(np.diff(gp) >= 0)
    o1, o2 = np.lexsort((gb, gp)), np.lexsort((br, pr))
    assert np.array_equal(gp[o1], pr[o2]) and np.array_equal(gb[o1], br[o2])
    hit = gb >= 0
    for j, x in enumerate(bp):
        v, nul = [c.cpu().numpy() for c in r["build"][j]]
        exp_null = ~hit | (bnull[gb] if j == 3 else False)
        assert np.array_equal(nul, exp_null)
        assert np.array_equal(v[~exp_null].view(np.uint8), x[gb[~exp_null]].view(np.uint8))
    assert np.array_equal(r["probe"][0][0].cpu().numpy(), pp[gp])
    t.free()


def test_one_long_chain_is_written_in_time(ctx):
    """One probe row of a key with 20,000 build rows: a row a round took 0.9 us a
    row, 18 ms; 0.1 us now.  0.4 us a row is allowed."""
    import torch
    nb, dup, n = 400_000, 20_000, 10_000
    bkey = np.arange(nb)
    bkey[:dup] = 7_000_000
    fk = dup + np.arange(n) % (nb - dup)
    fk[n // 2] = 7_000_000
    t = ctx.join_build(dev(bkey), build_payload=[dev(np.arange(nb)), dev(np.arange(nb) * 0.5)])
    fk = dev(fk)
    best = 1e9
    for _ in range(6):
        torch.cuda.synchronize()
        t0 = time.perf_counter()
        assert ctx.join_probe(t, fk, capacity=n + dup)["rows"] == n - 1 + dup
        best = min(best, time.perf_counter() - t0)
    t.free()
    assert best < 0.4e-6 * dup, best
