"""Lookups of one DAG on several streams and from several threads: its index is
made on the stream of the first lookup, and the others wait for it there."""
import os
import re
import threading

import numpy as np
import pytest

from cpvs_gb300 import scene

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "cpvs_gb300", "csrc")


def test_every_use_of_an_index_waits_for_it():
    with open(os.path.join(CSRC, "capi.cu")) as f:
        text = re.sub(r"//[^\n]*", "", f.read())
    for name in ("ensure_tops", "ensure_grid_top"):
        body = text[re.search(r"void %s\([^;{]*\{" % name, text).start():]
        body = body[:body.index("\n}\n")]
        assert body.index("index_mutex") < body.index("make_") < body.index("await_indices("), name
    for name in ("make_tops", "make_grid_top"):
        body = text[re.search(r"void %s\([^;{]*\{" % name, text).start():]
        assert "indexed_all(" in body[:body.index("\n}\n")], name


@pytest.fixture(scope="module")
def case(cp):
    import torch
    n = 1024
    d = scene.rasterise(scene.make_scene(n, 0.9, 60, 8, seed=4))
    q = scene.ndc_queries_mixed(d, 1 << 17, 9)
    return d, q, torch.from_numpy(q).cuda(), cp.CompressedShadow.from_depth(d).lookup_ndc(q)


def bits(cp, words, count):
    return cp.unpack_bits(words.cpu().numpy().view(np.uint32), count)


@pytest.mark.gpu
@pytest.mark.parametrize("kind", ["ndc", "voxel", "multi", "grid", "evaluate"])
def test_first_lookups_on_two_streams(cp, oracle, case, kind):
    """The index's making is held up on the first stream; a lookup on the second
    one, after a finished build, has to answer as ever."""
    import torch
    d, q, pts, want = case
    ctx = cp.Context(0)
    sh = cp.CompressedShadow.from_depth(d, ctx=ctx)
    lookup = {"ndc": lambda s: sh.lookup_ndc(pts, stream=s),
              "multi": lambda s: cp.lookup_ndc_multi([sh], torch.zeros(len(q), dtype=torch.int32, device="cuda"), pts,
                                                     stream=s)}.get(kind)
    if kind == "voxel":
        vox = ((pts + 1) * 0.5 * (d.shape[0] - 1)).int()
        want = oracle.lookup_voxel(sh.get_dag(), 11, True, vox.cpu().numpy()) if hasattr(oracle, "lookup_voxel") else \
            bits(cp, cp.CompressedShadow.from_depth(d).lookup_voxel(vox), len(q))
        lookup = lambda s: sh.lookup_voxel(vox, stream=s)  # noqa: E731
    if kind in ("grid", "evaluate"):
        grid = cp.CompressedShadowContainer.of(sh)
        grid.copy_to_gpu()
        pos = pts.view(256, -1, 3)
        lookup = (lambda s: grid.lookup_ndc(pts, stream=s)) if kind == "grid" else \
            (lambda s: grid.evaluate(pos, np.eye(4, dtype=np.float32), stream=s))
    a, b = torch.cuda.Stream(), torch.cuda.Stream()
    ctx.set_option(ctx.OPT_LOOKUP_QUERIES_PER_THREAD, 1)  # no timing of variants, which waits
    torch.cuda.synchronize()
    with torch.cuda.stream(a):
        torch.cuda._sleep(50_000_000)  # some tens of ms
    first = lookup(a)
    for _ in range(3):
        second = lookup(b)
        with torch.cuda.stream(b):
            got = (second.flatten() // 255).cpu().numpy() if kind == "evaluate" else bits(cp, second, len(q))
        assert np.array_equal(got, want), kind
    torch.cuda.synchronize()
    assert torch.equal(first, second)
    assert torch.equal(lookup(b), second) and torch.equal(lookup(a), second)


@pytest.mark.gpu
def test_a_second_streams_lookup_beside_another_threads_capture(cp, case):
    """The question whether an index is done, while another thread records a
    graph: the lookup answers and the recording goes on."""
    import torch
    d, q, pts, want = case
    ctx = cp.Context(0)
    ctx.set_option(ctx.OPT_LOOKUP_QUERIES_PER_THREAD, 1)
    sh = cp.CompressedShadow.from_depth(d, ctx=ctx)
    out = torch.zeros(len(q) // 32, dtype=torch.int32, device="cuda")
    a, b, c = (torch.cuda.Stream() for _ in range(3))
    x = torch.ones(64, device="cuda")
    torch.cuda.synchronize()
    sh.lookup_ndc(pts, out=out, stream=a)
    a.synchronize()
    recording, asked, graph = threading.Event(), threading.Event(), torch.cuda.CUDAGraph()

    def record():
        with torch.cuda.graph(graph, stream=c):
            x.add_(1)
            recording.set()
            asked.wait(20)
            x.add_(1)

    t = threading.Thread(target=record)
    t.start()
    assert recording.wait(20)
    try:
        sh.lookup_ndc(pts, out=out, stream=b)
    finally:
        asked.set()
        t.join()
    torch.cuda.synchronize()
    assert np.array_equal(bits(cp, out, len(q)), want)
    graph.replay()
    torch.cuda.synchronize()
    assert float(x[0]) == 3.0


@pytest.mark.gpu
def test_first_lookups_of_several_threads(cp, case):
    import torch
    d, q, pts, want = case
    ctx = cp.Context(0)
    ctx.set_option(ctx.OPT_LOOKUP_QUERIES_PER_THREAD, 2)
    for trial in range(4):
        sh = cp.CompressedShadow.from_depth(d, ctx=ctx)
        torch.cuda.synchronize()
        got, start = [None] * 6, threading.Barrier(6)

        def work(k):
            s = torch.cuda.Stream()
            start.wait()
            out = sh.lookup_ndc(pts, stream=s)
            s.synchronize()
            got[k] = bits(cp, out, len(q))

        threads = [threading.Thread(target=work, args=(k,)) for k in range(6)]
        for t in threads:
            t.start()
        for t in threads:
            t.join()
        for k, g in enumerate(got):
            assert g is not None and np.array_equal(g, want), (trial, k)
