"""Maps denser than the flat one that made the plan, where the leaf level and
the levels above it run over every SM: the level that overflows (the leaves
alone, or level 3 and the leaves) cuts its nodes' children at its last place,
the column pass finds no room for its runs, and the build is planned again once.
DAG words against the oracle's."""
import numpy as np
import pytest

FLAT = 0.4


def band(n, lo, hi, seed, cells=None):
    """Depths over the voxels [lo, hi) of a height of n, a random one per texel
    (or per square of cells x cells texels, across the leaf columns' borders)."""
    v = np.random.default_rng(seed).uniform(lo + 0.5, hi - 0.5, (n, n)).astype(np.float32) / np.float32(n)
    if cells:
        v = np.ascontiguousarray(v[::cells, ::cells].repeat(cells, 0).repeat(cells, 1)[:n, :n])
    return v


@pytest.mark.gpu
@pytest.mark.parametrize("n, spread, cells", [(1024, 16, None), (1024, 16, 12), (1024, 80, None), (1024, 300, 12),
                                              (2048, 16, 12), (2048, 32, 12), (2048, 100, 12)])
def test_denser_leaf_levels_match_oracle(cp, oracle, n, spread, cells):
    flat = np.full((n, n), FLAT, np.float32)
    # 16 voxels: the z-range of the flat map's level-3 nodes (32: level 4's)
    lo = int(FLAT * n) // max(16, spread & 32) * max(16, spread & 32)
    want = oracle.build(flat).dag
    for trial in range(2):
        ctx = cp.Context(0)
        ctx.set_option(ctx.OPT_BUILD_CLUSTER_CAP, 2048)
        ctx.set_option(ctx.OPT_BUILD_INSERT_WAVES, 1)
        dense = band(n, lo, lo + spread, trial, cells)
        for replans, d, w in ((0, flat, want), (1, dense, oracle.build(dense).dag), (0, flat, want)):
            sh = cp.CompressedShadow.from_depth(d, ctx=ctx)
            assert np.array_equal(sh.get_dag(), w), trial
            assert (ctx.last_build()["replans"] > 0) == (replans > 0), trial
