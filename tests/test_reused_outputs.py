"""NULL maps returned over output columns that a later call writes again are the
caller's own: a map kept from the first call does not change with the second."""
import numpy as np
import pytest

from ghive_b200 import abi


def test_maps_are_copies_unless_the_outputs_are_fresh():
    from ghive_b200.ops import _Outs
    o = _Outs([abi.INT, abi.DOUBLE], 4, "cpu")
    for _, null in o.cols:
        null.copy_(null.new_tensor([1, 0, 1, 1]))
    kept, view = o.rows(3), o.rows(3, fresh=True)
    for _, null in o.cols:
        null.zero_()
    for (_, a), (_, b) in zip(kept, view):
        assert a.tolist() == [True, False, True] and b.tolist() == [False, False, False]


@pytest.mark.gpu
def test_maps_kept_over_calls_that_reuse_their_outputs():
    import torch
    from ghive_b200.ops import Context, _Outs
    n = 5000
    g = np.random.default_rng(2)
    x = torch.from_numpy(g.integers(0, 100, n)).cuda()
    null = [torch.from_numpy(g.random(n) < p).cuda() for p in (0.3, 0.7)]
    with Context(0) as ctx:
        outs = _Outs([abi.LONG], n, "cuda:0")
        first = ctx.filter(None, [(x, null[0])], outs=outs)[0][0][1]
        second = ctx.filter(None, [(x, null[1])], outs=outs)[0][0][1]
        assert torch.equal(first, null[0]) and torch.equal(second, null[1])
        order = torch.argsort(x, stable=True)
        souts = (_Outs([abi.LONG], n, "cuda:0"), _Outs([abi.LONG], n, "cuda:0"))
        first = ctx.sort([x], payload=[(x, null[0])], outs=souts)[1][0][1]
        second = ctx.sort([x], payload=[(x, null[1])], outs=souts)[1][0][1]
        assert torch.equal(first, null[0][order]) and torch.equal(second, null[1][order])
        t = ctx.join_build(torch.arange(100, device="cuda"))
        jouts = (_Outs([], n, "cuda:0"), _Outs([abi.LONG], n, "cuda:0"), None, None,
                 torch.empty(1, dtype=torch.int64, device="cuda"))
        first = ctx.join_probe(t, x, probe_payload=[(x, null[0])], capacity=n, outs=jouts)["probe"][0][1]
        second = ctx.join_probe(t, x, probe_payload=[(x, null[1])], capacity=n, outs=jouts)["probe"][0][1]
        assert torch.equal(first, null[0]) and torch.equal(second, null[1])
        t.free()
        # a batch writes the same outputs at each launch
        one, mask = torch.zeros(n, dtype=torch.int64, device="cuda"), torch.ones(n, dtype=torch.uint8, device="cuda")
        b = ctx.batch_groupby([(None, [one, (x, mask)], 4, 4)], [0], [(abi.MAX, 1)], autotune=False)
        b.launch()
        ctx.sync()
        first = b.results(0)[1][0][1]
        mask.zero_()
        b.launch()
        ctx.sync()
        second = b.results(0)[1][0][1]
        assert first.tolist() == [True] and second.tolist() == [False]
        b.free()
