"""A lookup over many DAGs that is refused makes no index for them."""
import ctypes as C

import numpy as np
import pytest

from cpvs_gb300 import scene


@pytest.mark.gpu
def test_refused_multi_lookups_hold_nothing(cp):
    import torch
    lib = cp.load_library()
    ctx = cp.Context(0)
    d = scene.rasterise(scene.make_scene(512, 0.9, 20, 2, seed=1))
    h = cp.MinMaxHierarchy(d, ctx=ctx)
    for count in (3, 70):  # the table in the launch's parameters, and in memory
        shadows = cp.CompressedShadow.create_batch([h], [(0, 0, 1)] * count)
        tab = (C.c_void_p * count)(*[s.handle for s in shadows])
        pts, ids = torch.zeros((64, 3), device="cuda"), torch.zeros(64, dtype=torch.int32, device="cuda")
        out = torch.zeros(2, dtype=torch.int32, device="cuda")
        held = ctx.bytes_in_use()
        for xyz, bits, n in ((None, out.data_ptr(), 64), (pts.data_ptr(), None, 64), (pts.data_ptr(), out.data_ptr(), 1 << 40)):
            status = lib.cpvs_lookup_ndc_multi(tab, count, ids.data_ptr(), xyz, n, bits, cp.IO_DEVICE, None)
            assert status != 0 and ctx.bytes_in_use() == held, n
        # (no points: nothing to do)
        assert lib.cpvs_lookup_ndc_multi(tab, count, ids.data_ptr(), None, 0, None, cp.IO_DEVICE, None) == 0
        assert ctx.bytes_in_use() == held
        got = cp.lookup_ndc_multi(shadows, ids, pts, out=out)
        assert np.array_equal(cp.unpack_bits(got.cpu().numpy().view(np.uint32), 64), shadows[0].lookup_ndc(pts.cpu().numpy()))
