"""Group-bys on a card whose free memory holds their global tables at a load factor
of 0.5 and not at 0.25: they run as they do with memory to spare."""
import numpy as np
import pytest

from ghive_b200 import workloads

pytestmark = pytest.mark.gpu

MB = 1 << 20


def columns(n, groups, seed):
    import torch
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    k = torch.cat([torch.arange(groups, device="cuda"),
                   torch.randint(0, groups, (n - groups,), generator=g, device="cuda")])
    return [workloads.mix64_torch(k), torch.randint(1, 51, (n,), generator=g, device="cuda"),
            torch.rand(n, generator=g, device="cuda", dtype=torch.float64),
            torch.zeros(n, device="cuda", dtype=torch.int32)]


def ordered(ks, vs):
    import torch
    o = torch.argsort(ks[0][0])
    return [x[o].cpu().numpy() for x, _ in ks + vs]


def same(a, b):
    return all(np.array_equal(x, y) if x.dtype != np.float64 else np.all(np.abs(x - y) <= 1e-12 * np.abs(x))
               for x, y in zip(a, b))


# 1M groups of the fact aggregates: records of 64 bytes, 2M slots (134 MB) at a
# load factor of 0.5 and 4M (268 MB) at 0.25
def test_group_by_with_room_for_the_smaller_table():
    import torch
    from ghive_b200.ops import Context
    n = groups = 1_000_000
    cols = columns(n, groups, 1)
    args = (workloads.fact_predicate(), cols, [0], workloads.AGGS_FACT)
    with Context(0) as ctx:
        ks, vs, m = ctx.filter_groupby(*args, capacity=groups, max_groups=groups)
        assert m == groups
        exp = ordered(ks, vs)
        del ks, vs   # their blocks serve the call below
    with Context(0) as ctx:
        torch.cuda.synchronize()
        fill = torch.empty(torch.cuda.mem_get_info()[0] - 210 * MB, dtype=torch.uint8, device="cuda")
        try:
            for _ in range(2):   # the second keeps the first one's table
                ks = vs = None
                ks, vs, m = ctx.filter_groupby(*args, capacity=groups, max_groups=groups)
        finally:
            del fill
            torch.cuda.empty_cache()
        assert m == groups and same(ordered(ks, vs), exp)


def test_batch_with_room_for_the_smaller_tables():
    import torch
    from ghive_b200.ops import Context
    n = groups = 1_000_000
    insts = [(workloads.fact_predicate(), columns(n, groups, s), groups, groups) for s in (2, 3)]

    def run(ctx, fill):
        held = torch.empty(torch.cuda.mem_get_info()[0] - fill, dtype=torch.uint8, device="cuda") if fill else None
        try:
            b = ctx.batch_groupby(insts, [0], workloads.AGGS_FACT, autotune=False)
        finally:
            del held
            torch.cuda.empty_cache()
        b.launch()
        ctx.sync()
        out = [ordered(*b.results(i)[:2]) for i in range(2)]
        lf = [c["load_factor"] for c in b.describe()["classes"]]
        b.free()
        return out, lf

    with Context(0) as ctx:
        exp, lf = run(ctx, 0)
        assert lf == [0.25]
    with Context(0) as ctx:
        torch.cuda.empty_cache()
        got, lf = run(ctx, 500 * MB)   # outputs up to 160 MB, tables 268 or 537
        assert lf == [0.5]
        assert all(same(a, b) for a, b in zip(exp, got))
