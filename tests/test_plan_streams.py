"""A plan's builds on several streams: what one build leaves for the next is
ordered by the plan's event alone, so everything that it leaves comes before
the event's last record."""
import os
import re

import numpy as np
import pytest

from cpvs_gb300 import scene

SOURCE = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "cpvs_gb300", "csrc", "build.cu")


def body(name):
    """The text of the function `name`, comments left out."""
    with open(SOURCE) as f:
        text = re.sub(r"//[^\n]*", "", f.read())
    text = text[re.search(r"^cpvs_status %s\([^;{]*\{" % name, text, re.M).start():]
    return text[:text.index("\n}\n")]


def test_the_level_table_is_copied_before_the_plans_event():
    b = body("build_dags")
    assert b.rindex("cudaMemcpyAsync(P->lvt") < b.rindex("cudaEventRecord(P->done")


@pytest.mark.gpu
@pytest.mark.parametrize("n", [256, 1024])
def test_builds_of_one_shape_on_two_streams_match_oracle(cp, oracle, n):
    """Fixed launch shapes: no tuning between a plan's first build, which sizes
    the hash tables, and the second one's."""
    import torch
    maps = [scene.rasterise(scene.make_scene(n, 0.9, 12 + 9 * k, 3 * k, seed=k)) for k in range(4)]
    want = [oracle.build(d).dag for d in maps]
    dev = [torch.from_numpy(d).cuda() for d in maps]
    torch.cuda.synchronize()
    streams = [torch.cuda.Stream() for _ in range(2)]
    for trial in range(4):
        ctx = cp.Context(0)
        ctx.set_option(ctx.OPT_BUILD_CLUSTER_CAP, 2048)
        ctx.set_option(ctx.OPT_BUILD_INSERT_WAVES, 1)
        got = [cp.CompressedShadow.from_depth(d, ctx=ctx, stream=streams[i % 2]) for i, d in enumerate(dev)]
        for i, sh in enumerate(got):
            assert np.array_equal(sh.get_dag(stream=streams[i % 2]), want[i]), (trial, i)
