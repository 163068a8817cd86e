"""The shared slots of a batch that is not tuned: as many as the instances'
numbers of groups need, so that 1500 groups keep their rows out of the global
tables.  Results equal each instance's own call."""
import numpy as np
import pytest

from ghive_b200 import abi, workloads

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    from ghive_b200.ops import Context
    c = Context(0)
    yield c
    c.close()


# groups of each instance (60,000 rows apiece; None: not stated, half the rows as capacity) and the slots
@pytest.mark.parametrize("groups,slots", [
    ([100] * 4, 256), ([700] * 4, 1024), ([1024] * 4, 1024), ([1025] * 4, 2048), ([2048] * 4, 2048),
    ([2049] * 4, 1024), ([20_000] * 4, 1024), ([1500] * 3 + [3000], 2048), ([1500] * 2 + [3000] * 2, 1024),
    ([1500] + [700] * 3, 2048), ([1500] + [700] * 4, 1024), ([1500] + [100] * 5, 2048), ([None] * 4, 1024)])
def test_shared_slots_of_an_untuned_batch(ctx, groups, slots):
    import torch
    g = np.random.default_rng(8)
    n, insts, exp = 60_000, [], []
    pred = workloads.fact_predicate(2270)
    for m in groups:
        k = g.integers(0, m or 1500, n)
        cols = [torch.from_numpy(c).cuda() for c in (k, g.integers(1, 51, n), g.integers(90000, 10500001, n) / 100.0,
                                                     g.integers(0, 2526, n, dtype=np.int32))]
        insts.append((pred, cols, m or n // 2, m or 0))
        exp.append(ctx.filter_groupby(pred, cols, [0], workloads.AGGS_FACT, capacity=n))
    b = ctx.batch_groupby(insts, [0], workloads.AGGS_FACT, autotune=False)
    assert max(c["smem_slots"] for c in b.describe()["classes"]) == slots
    b.launch()
    ctx.sync()
    for i, (ks, vs, m) in enumerate(exp):
        bk, bv, bm = b.results(i)
        assert bm == m
        o1, o2 = torch.argsort(ks[0][0]), torch.argsort(bk[0][0])
        for (x, _), (y, _) in zip(ks + vs, bk + bv):
            x, y = x[o1].cpu().numpy(), y[o2].cpu().numpy()
            assert np.array_equal(x, y) if x.dtype != np.float64 else np.all(np.abs(x - y) <= 1e-12 * np.abs(x))
    b.free()
