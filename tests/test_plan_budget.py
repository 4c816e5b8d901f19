"""A plan that has to grow and finds no room for it: the build fails with the
budget's error, and the next builds of that shape work as if it had not been."""
import numpy as np
import pytest

from cpvs_gb300 import scene


def test_a_plan_that_cannot_grow_leaves_the_cache():
    import os
    import re
    with open(os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "cpvs_gb300", "csrc", "build.cu")) as f:
        text = re.sub(r"//[^\n]*", "", f.read())
    text = text[re.search(r"^cpvs_status build_dags\([^;{]*\{", text, re.M).start():]
    grow = text[text.index("plan_allocate("):]
    assert "plan_drop(ctx, P)" in grow[:grow.index("return r;")]


@pytest.mark.gpu
@pytest.mark.parametrize("leafmasks", [True, False])
def test_builds_after_one_without_room_to_grow(cp, oracle, leafmasks):
    n = 256 if leafmasks else 128
    sparse = [scene.rasterise(scene.make_scene(n, 0.9, 2, 0, seed=k)) for k in range(2)]
    dense = np.random.default_rng(1).random((n, n), np.float32)
    ctx = cp.Context(0)

    def same(d):
        got = cp.CompressedShadow.from_depth(d, leafmasks=leafmasks, ctx=ctx)
        return np.array_equal(got.get_dag(), oracle.build(d, leafmasks=leafmasks).dag)

    assert same(sparse[0])
    ctx.set_budget(ctx.bytes_in_use() + (2 << 20))
    for _ in range(2):
        with pytest.raises(cp.CpvsError, match="budget"):
            cp.CompressedShadow.from_depth(dense, leafmasks=leafmasks, ctx=ctx)
        assert same(sparse[1])
    ctx.set_budget(0)
    assert same(dense) and same(sparse[0])
