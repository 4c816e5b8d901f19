"""The memory that indices deeper than their DAGs' sizes allow may hold: 1 GiB a
context, whatever the number of DAGs whose first lookup is a large one."""
import numpy as np
import pytest


@pytest.mark.gpu
def test_deep_indices_are_bounded(cp):
    import torch
    n, count, limit = 2048, 20, 1 << 30
    gen = torch.Generator("cuda").manual_seed(1)
    pts = torch.rand((1 << 25, 3), device="cuda", generator=gen) * 2 - 1
    depth = torch.full((n, n), 0.4, device="cuda")
    depth[100:900, 300:1500] = 0.25
    torch.cuda.synchronize()
    ctx = cp.Context(0)
    h = cp.MinMaxHierarchy(depth, ctx=ctx, borrow=True)
    for again in range(2):  # the second time the first ones' memory is there again
        shadows = cp.CompressedShadow.create_batch([h], [(0, 0, 1)] * count)
        before = ctx.bytes_in_use()
        want = shadows[0].lookup_ndc(pts)
        deep = ctx.bytes_in_use() - before
        assert deep == 64 << 20  # a cell per two points
        for sh in shadows[1:]:
            assert torch.equal(sh.lookup_ndc(pts), want)
        held = ctx.bytes_in_use() - before
        assert limit - deep < held <= limit + count * (64 << 10)
        del shadows, sh
    ids = torch.zeros(pts.shape[0], dtype=torch.int32, device="cuda")
    shadows = cp.CompressedShadow.create_batch([h], [(0, 0, 1)] * count)
    before = ctx.bytes_in_use()
    got = cp.lookup_ndc_multi(shadows, ids, pts)
    assert torch.equal(got, want)
    assert ctx.bytes_in_use() - before <= limit + count * (64 << 10)
