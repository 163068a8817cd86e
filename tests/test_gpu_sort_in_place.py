"""ORDER BY whose outputs are its own input columns: a key of at most 64 bits,
alone or with one payload that carries no NULL map, sorted in place."""
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


def outs_over(cols, types):
    """Output columns that are these device columns."""
    from ghive_b200.ops import _Outs
    o = _Outs(types, 1, "cuda:0", with_nulls=False)
    for i, c in enumerate(cols):
        o.cols[i] = (c, None)
        o.arr[i].data = c.data_ptr()
    return o


@pytest.mark.parametrize("n", [1000, 4000, 8192, 8193, 100_000])
@pytest.mark.parametrize("bits", [12, 48])
def test_sorted_in_place(ctx, n, bits):
    import torch
    g = np.random.default_rng(n + bits)
    for _ in range(5):
        k, d = g.integers(0, 1 << bits, n), g.integers(0, 9, n, dtype=np.int32)
        x = g.random(n)
        perm = oracle.sort_perm([d, k], threads=8)
        dk, dd, dx = (torch.from_numpy(a).cuda() for a in (k, d, x))
        ctx.sort([dd, dk], payload=[dx], outs=(outs_over([dd, dk], [abi.INT, abi.LONG]), outs_over([dx], [abi.DOUBLE])))
        assert np.array_equal(dd.cpu().numpy(), d[perm])
        assert np.array_equal(dk.cpu().numpy(), k[perm])
        assert np.array_equal(dx.cpu().numpy(), x[perm])
