"""The NULL map of a STRING column that a filter projects: a row is NULL when
its pair starts below 0, whatever decides that the row passes."""
import numpy as np
import pytest

from ghive_b200 import abi

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


@pytest.mark.parametrize("n", [1, 2047, 50_000])
@pytest.mark.parametrize("cut", [0, 40, 100])
def test_null_map_of_a_projected_string(ctx, n, cut):
    g = np.random.default_rng(n + cut)
    null = g.random(n) < 0.3
    start = np.arange(n, dtype=np.int32) * 3
    pairs = np.stack([np.where(null, -1, start), np.where(null, -1, start + 3)], 1).astype(np.int32)
    chars = g.integers(97, 123, 3 * n, dtype=np.uint8)
    d = g.integers(0, 100, n, dtype=np.int32)
    sel = np.flatnonzero(d < cut)
    s = ("string", dev(chars), dev(pairs.reshape(-1)))
    (sv, sn), (dv, dn) = ctx.filter(abi.Pred.leaf(abi.FILTER_LT, 1, a=cut), [s, dev(d)], proj=[0, 1])[0]
    assert np.array_equal(sv.cpu().numpy().reshape(-1, 2), pairs[sel])
    assert np.array_equal(sn.cpu().numpy(), null[sel])
    assert np.array_equal(dv.cpu().numpy(), d[sel]) and not dn.any().item()
