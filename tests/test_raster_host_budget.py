"""Triangles rasterised into host memory by a context whose budget leaves no room
for the window's scratch: the pixels are lowered where they lie."""
import numpy as np
import pytest

from cpvs_gb300 import scene


@pytest.mark.gpu
@pytest.mark.parametrize("n, cells, window", [(64, 5, None), (256, 24, (31, 17, 130, 77)), (512, 3, None)])
def test_host_output_without_room_for_the_window(cp, n, cells, window):
    t = scene.terrain_triangles(cells, 3)
    want = scene.rasterise_triangles(t, n, 0.9)
    x0, y0, w, h = window or (0, 0, n, n)
    want = want[y0:y0 + h, x0:x0 + w]
    ctx = cp.Context(0)
    for budget in (0, 1, 4 * w * h, 2 << 20):  # none, no room at all, for the window alone, for the triangles' list too
        ctx.set_budget(budget)
        got = cp.raster_triangles(t, n, 0.9, x0=x0, y0=y0, w=w, h=h, ctx=ctx)
        assert np.array_equal(got.view(np.uint32), want.view(np.uint32)), budget
        assert ctx.bytes_in_use() == 0
