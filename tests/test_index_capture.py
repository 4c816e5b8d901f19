"""A DAG's first lookup recorded in a graph: the graph's memory and work are
there when it runs, so no index is made in it, and lookups outside it answer as
ever before, between and after its runs."""
import os
import re

import numpy as np
import pytest

from cpvs_gb300 import scene

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "cpvs_gb300", "csrc")


def test_no_index_is_made_in_a_capture():
    with open(os.path.join(CSRC, "capi.cu")) as f:
        text = re.sub(r"//[^\n]*", "", f.read())
    for name in ("void make_tops", "void make_grid_top", "int lookup_qpt"):
        body = text[re.search(name + r"\([^;{]*\{", text).start():]
        body = body[:body.index("\n}\n")]
        first = body.index("capturing(st)")
        assert all(first < body.index(c) for c in ("alloc(", "tune_lookup(") if c in body), name


def test_no_recorded_copy_of_a_calls_own_table():
    with open(os.path.join(CSRC, "capi.cu")) as f:
        text = re.sub(r"//[^\n]*", "", f.read())
    body = text[re.search(r"cpvs_status cpvs_lookup_ndc_multi\([^;{]*\{", text).start():]
    assert "cudaMemcpyAsync" not in body[:body.index("\n}\n")]
    with open(os.path.join(CSRC, "lookup.cu")) as f:
        text = f.read()
    body = text[re.search(r"cpvs_status put_multi_table\([^;{]*\{", text).start():]
    assert body.index("if (!capturing(st))") < body.index("cudaMemcpyAsync")


@pytest.mark.gpu
@pytest.mark.parametrize("count", [64, 65, 150])
def test_many_dags_in_a_graph(cp, count):
    """A table larger than a launch's parameters: it is the graph's, whatever
    becomes of the memory that the recording call had it in."""
    import torch
    ctx = cp.Context(0)
    maps = [scene.rasterise(scene.make_scene(64, 0.9, 3 + k % 7, 1, seed=k)) for k in range(10)]
    hs = cp.MinMaxHierarchy.create_batch(maps, ctx=ctx)
    shadows = cp.CompressedShadow.create_batch(hs, [(k % 10, 0, 1) for k in range(count)])
    g = torch.Generator("cuda").manual_seed(3)
    pts = torch.rand((1 << 15, 3), device="cuda", generator=g) * 2 - 1
    ids = torch.randint(count, (1 << 15,), device="cuda", generator=g, dtype=torch.int32)
    want = cp.lookup_ndc_multi(shadows, ids, pts)
    out = torch.zeros_like(want)
    torch.cuda.synchronize()
    stream, graph = torch.cuda.Stream(), torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        cp.lookup_ndc_multi(shadows, ids, pts, out=out, stream=stream)
    junk = [np.full(count * 10, 0x5A5A5A5A, np.uint32) for _ in range(64)]
    for _ in range(2):
        out.zero_()
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(out, want)
    del junk


@pytest.mark.gpu
@pytest.mark.parametrize("kind", ["ndc", "multi", "grid", "evaluate"])
def test_first_lookup_in_a_graph(cp, oracle, kind):
    import torch
    n = 512
    d = scene.rasterise(scene.make_scene(n, 0.9, 40, 4, seed=7))
    q = scene.ndc_queries_mixed(d, 1 << 16, 5)
    want = cp.CompressedShadow.from_depth(d).lookup_ndc(q)
    pts = torch.from_numpy(q).cuda()
    ctx = cp.Context(0)
    sh = cp.CompressedShadow.from_depth(d, ctx=ctx)
    ids = torch.zeros(len(q), dtype=torch.int32, device="cuda")
    u8 = torch.zeros((128, len(q) // 128), dtype=torch.uint8, device="cuda")
    words = torch.zeros(len(q) // 32, dtype=torch.int32, device="cuda")
    pos = pts.view(128, -1, 3)
    if kind in ("grid", "evaluate"):
        grid = cp.CompressedShadowContainer.of(sh)
        grid.copy_to_gpu()
    run = {"ndc": lambda s, o: sh.lookup_ndc(pts, out=o, stream=s),
           "multi": lambda s, o: cp.lookup_ndc_multi([sh], ids, pts, out=o, stream=s),
           "grid": lambda s, o: grid.lookup_ndc(pts, out=o, stream=s),
           "evaluate": lambda s, o: grid.evaluate(pos, np.eye(4, dtype=np.float32), out=o, stream=s)}[kind]
    out = u8 if kind == "evaluate" else words

    def same(o):
        torch.cuda.synchronize()
        got = (o.flatten() // 255).cpu().numpy() if kind == "evaluate" else \
            cp.unpack_bits(o.cpu().numpy().view(np.uint32), len(q))
        return np.array_equal(got, want)

    # the kernels' code is loaded before the capture
    other = cp.CompressedShadow.from_depth(d)
    other.lookup_ndc(pts)
    cp.lookup_ndc_multi([other], ids, pts)
    g2 = cp.CompressedShadowContainer.of(other)
    g2.copy_to_gpu()
    g2.lookup_ndc(pts)
    g2.evaluate(pos, np.eye(4, dtype=np.float32))
    torch.cuda.synchronize()
    held = ctx.bytes_in_use()
    stream, graph = torch.cuda.Stream(), torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        run(stream, out)
    assert ctx.bytes_in_use() == held
    eager = torch.zeros_like(out)
    run(None, eager)  # before the graph's first run: an index of its own
    assert same(eager)
    for _ in range(2):
        out.zero_()
        graph.replay()
        assert same(out)
        eager.zero_()
        run(None, eager)
        assert same(eager)


@pytest.mark.gpu
def test_objects_used_in_a_graph_are_destroyed(cp, oracle):
    """An object whose last use was recorded in a capture: its release waits for
    nothing of the capture and leaves no error behind for the next call."""
    import torch
    n = 256
    d = scene.rasterise(scene.make_scene(n, 0.9, 20, 4, seed=2))
    want = oracle.build(d).dag
    q = scene.ndc_queries_mixed(d, 1 << 12, 5)
    pts = torch.from_numpy(q).cuda()
    out = torch.zeros(len(q) // 32, dtype=torch.int32, device="cuda")
    ctx = cp.Context(0)
    ids = torch.zeros(len(q), dtype=torch.int32, device="cuda")
    for trial in range(3):
        sh = cp.CompressedShadow.from_depth(d, ctx=ctx)
        sh.lookup_ndc(pts)
        torch.cuda.synchronize()
        stream, graph = torch.cuda.Stream(), torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=stream):
            sh.lookup_ndc(pts, out=out, stream=stream)
            cp.lookup_ndc_multi([sh], ids, pts, out=out, stream=stream)
        graph.replay()
        torch.cuda.synchronize()
        del graph, sh
        again = cp.CompressedShadow.from_depth(d, ctx=ctx)
        assert np.array_equal(again.get_dag(), want)
        del again
