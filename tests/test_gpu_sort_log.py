"""A sort's log line tells the radix passes it launched and whether a finish sorts
the rest, which its number of kernels alone does not: five leading digits and the
two finish kernels are as many as seven digits."""
import json

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_passes_and_finish(tmp_path):
    import torch

    from ghive_b200.ops import Context
    g = np.random.default_rng(6)
    n = 100_000
    far = g.integers(0, 1 << 39, n)          # the first 23 of 62 bits tell nothing
    far[7] = (1 << 62) - 1
    hot = g.integers(0, 1 << 52, n)
    hot[:n // 2] = 77                        # half of the rows share a key
    far, hot, few = (torch.from_numpy(x).cuda() for x in (far, hot, g.integers(0, 1000, 5000)))
    path = tmp_path / "sorts.jsonl"
    kernels = []
    with Context(0) as ctx:
        ctx.set_log(path)
        for k in (far, hot, few):
            before = ctx.launches
            ctx.sort([k], payload=[k])
            kernels.append(ctx.launches - before)
    lines = [json.loads(x) for x in path.read_text().splitlines()]
    assert [(x.get("passes"), x.get("finish")) for x in lines] == [(5, 1), (7, 0), (None, None)]
    assert kernels == [10, 10, 1]
