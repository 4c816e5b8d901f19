"""Depth maps that begin off a 16-byte boundary (a contiguous view into a larger
buffer): the kernels read maps in 16-byte loads, so such a map is copied first,
wherever a map enters."""
import ctypes as C
import os
import re

import numpy as np
import pytest

from cpvs_gb300 import scene

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "cpvs_gb300", "csrc")


@pytest.mark.parametrize("name, function", [("capi.cu", "hierarchy_create"), ("capi.cu", "cpvs_hierarchy_create_batch"),
                                            ("build.cu", "cpvs_shadow_build_noalloc")])
def test_every_entry_of_a_map_asks_for_its_alignment(name, function):
    with open(os.path.join(CSRC, name)) as f:
        text = f.read()
    text = text[re.search(r"cpvs_status %s\([^;{]*\{" % function, text).start():]
    assert "aligned16(" in text[:text.index("\n}\n")]


def view(d, offset, device, pinned=False):
    """`d` in memory `offset` floats past a 16-byte boundary."""
    import torch
    if not device and not pinned:
        buf = np.empty(d.size + 8, np.float32)
        at = (-buf.ctypes.data // 4) % 4 + offset
        v = buf[at:at + d.size].reshape(d.shape)
        v[...] = d
        assert v.ctypes.data % 16 == 4 * offset
        return v
    buf = torch.empty(d.size + 8, dtype=torch.float32, pin_memory=pinned, device="cuda" if device else None)
    v = buf[offset:offset + d.size].view(*d.shape)
    v.copy_(torch.from_numpy(d))
    assert v.data_ptr() % 16 == 4 * offset
    return v


@pytest.mark.gpu
@pytest.mark.parametrize("n", [8, 16, 64, 256, 1024])
@pytest.mark.parametrize("offset", [1, 2, 3])
def test_unaligned_maps_match_oracle(cp, oracle, n, offset):
    d = scene.rasterise(scene.make_scene(n, 0.9, 10, 4, seed=n + offset))
    for leafmasks in (True, False):
        if not leafmasks and n > 64:
            continue
        want = oracle.build(d, leafmasks=leafmasks).dag
        for device, pinned in ((True, False), (False, False), (False, True)):
            m = view(d, offset, device, pinned)
            got = cp.CompressedShadow.from_depth(m, leafmasks=leafmasks)
            assert np.array_equal(got.get_dag(), want), (leafmasks, device, pinned)
            h = cp.MinMaxHierarchy(m, borrow=True) if device else cp.MinMaxHierarchy(m)
            m[...] = 0 if not device else m  # a host map may be reused on return
            got = cp.CompressedShadow.create(h, leafmasks=leafmasks)
            assert np.array_equal(got.get_dag(), want), (leafmasks, device, pinned)


@pytest.mark.gpu
@pytest.mark.parametrize("device", [True, False])
def test_unaligned_maps_of_a_batch_match_oracle(cp, oracle, device):
    maps = [scene.rasterise(scene.make_scene(n, 0.9, 10, 2, seed=n)) for n in (16, 64, 128, 512)]
    hs = cp.MinMaxHierarchy.create_batch([view(d, i % 4, device) for i, d in enumerate(maps)], borrow=device)
    for d, sh in zip(maps, cp.CompressedShadow.create_batch(hs, [(i, 0, 1) for i in range(len(maps))])):
        assert np.array_equal(sh.get_dag(), oracle.build(d).dag)


@pytest.mark.gpu
@pytest.mark.parametrize("n, leafmasks", [(8, True), (64, False), (64, True), (256, True)])
def test_unaligned_map_of_the_allocation_free_build(cp, oracle, n, leafmasks):
    import torch
    lib = cp.load_library()
    d = scene.rasterise(scene.make_scene(n, 0.9, 10, 2, seed=n))
    want = oracle.build(d, leafmasks=leafmasks).dag
    for offset in (0, 1, 2, 3):
        m = view(d, offset, True)
        out, words = torch.zeros(1 << 18, dtype=torch.int32, device="cuda"), C.c_uint64(0)
        status = lib.cpvs_shadow_build_noalloc(m.data_ptr(), n, 0, 1, 1 if leafmasks else 0, out.data_ptr(), out.numel(),
                                               C.byref(words), None)
        assert status == 0, lib.cpvs_last_error()
        assert np.array_equal(out[:words.value].cpu().numpy().view(np.uint32), want), offset
