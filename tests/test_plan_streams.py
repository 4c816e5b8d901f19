"""The order of a build's work over streams.  What one build of a plan leaves
for the next is ordered by the plan's event alone, so everything that it leaves
comes before the event's last record.  Within a build, a word that errors are
reported in is cleared before anything may report there."""
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


def test_the_leaf_branch_reports_in_a_word_of_its_own():
    """The results' region is cleared on the level chain's stream, beside the
    branch: what the branch reports lies in what its own stream cleared before,
    and the last kernel joins the two."""
    b = body("plan_enqueue")
    for launch in re.findall(r"launch_kernel\([^;]*k_leaf_(?:columns|classes)[^;]*;", b):
        assert not re.search(r"\berr\b", launch), launch
    assert b.index("P->lmeta + 4") < b.index("k_leaf_columns<true>")
    assert "lc.err" in b[b.index("k_layout"):]


@pytest.mark.gpu
@pytest.mark.parametrize("timing", [False, True])
def test_a_full_class_table_is_reported(cp, oracle, timing):
    """The same 8x8 texels in every column, whose few leaf classes size the
    table, then other ones in each column of a half and again in the other half:
    more classes than it holds, while no level outgrows the plan and the inner
    levels' tables suffice."""
    n = 256
    rng = np.random.default_rng(3)
    tile = rng.uniform(0.3, 0.42, (8, 8)).astype(np.float32)
    alike = np.tile(tile, (n // 8, n // 8))
    # each column's texels in another order: the same bounds, so the same nodes
    half = np.block([[rng.permutation(tile.ravel()).reshape(8, 8) for _ in range(n // 16)] for _ in range(n // 8)])
    other = np.concatenate([half, half], 1)
    ctx = cp.Context(0)
    ctx.enable_timing(timing)
    for k, d in enumerate((alike, np.ascontiguousarray(other))):
        sh = cp.CompressedShadow.from_depth(d, ctx=ctx)
        assert np.array_equal(sh.get_dag(), oracle.build(d).dag)
        assert ctx.last_build()["replans"] == k


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
