"""The work whose speed counts: what a program that uses this package has it
do, through the package's Python entry points, over the range of sizes it
meets in use.

  build    depth map -> resident shadow DAG (CompressedShadow.from_depth), its
           words in the program's own buffer (as the reference uploads them
           to the buffer its shader reads)
  lights   many lights of different map sides in one batch, then their first
           lookups (MinMaxHierarchy.create_batch + CompressedShadow.create_batch
           + lookup_ndc_multi)
  grid     a map cut into tiles and z-tiles, built as one container and
           looked up through it (CompressedShadowContainer.build + lookup_ndc)
  lookup   batched visibility of light-space points (lookup_ndc, lookup_voxel)
  multi    points spread over many resident DAGs (lookup_ndc_multi)
  frame    one rendered frame: evaluate a G-buffer, then shade it
  pcf      evaluate with a percentage-closer filter
  raster   a triangle mesh into a depth map (raster_triangles)

Scenes are a ground plane with boxes and spheres on it, as the package's own
benchmark uses, drawn here with torch so that `exact` needs nothing of the
package; box and sphere counts and extents are the benchmark's.
"""
import math

import numpy as np
import torch

import cpvs_gb300 as cp

DEV = "cuda"


def listed():
    return [
        # A small light (a spot or point light's face): nothing but launches
        # and dependent round trips.
        {"name": "build_256", "kind": "build", "n": 256, "boxes": 20, "spheres": 4, "host": False},
        # One ordinary shadow map; rebuilt when its light moves.
        {"name": "build_1024", "kind": "build", "n": 1024, "boxes": 40, "spheres": 0, "host": False},
        # The largest single map (the tile cap of the reference's renderer).
        {"name": "build_8192", "kind": "build", "n": 8192, "boxes": 500, "spheres": 64, "host": False},
        # End to end: the map in pinned host memory, the DAG words back in it.
        {"name": "build_host_4096", "kind": "build", "n": 4096, "boxes": 300, "spheres": 32, "host": True},
        # A scene's lights precomputed together (sides 256 .. 4096), then their
        # first lookups.
        {"name": "lights_16", "kind": "lights", "lights": 16, "lo": 8, "hi": 12, "points": 1 << 18},
        # An 8192^2 map as 4x4 tiles x 4 z-tiles (64 DAGs), then its first lookups.
        {"name": "grid_4x2048", "kind": "grid", "length": 4, "n": 2048, "points": 1 << 20},
        # A few voxels of one object asked for by a game loop: latency, ragged.
        {"name": "lookup_voxel_1000", "kind": "lookup", "n": 1024, "points": 1000, "voxel": True},
        # Bulk visibility against the largest map (light baking): half of the
        # points on the surface, half anywhere in the volume.
        {"name": "lookup_8192_2e26", "kind": "lookup", "n": 8192, "points": 1 << 26, "voxel": False},
        # Points of a frame or a bake that several lights reach.
        {"name": "multi_16", "kind": "multi", "lights": 16, "lo": 8, "hi": 12, "points": (1 << 22) + 3},
        # A 4K frame against the largest map.
        {"name": "frame_2160p", "kind": "frame", "n": 8192, "width": 3840, "height": 2160},
        # A filtered (soft-edged) frame at 1080p.
        {"name": "pcf3_1080p", "kind": "pcf", "n": 4096, "width": 1920, "height": 1080, "filter": 3},
        # A terrain mesh of half a million triangles under the light.
        {"name": "raster_512x512", "kind": "raster", "cells": 512, "n": 2048, "width": 2048, "height": 2048},
    ]


def _log2(rng, lo, hi):
    return 1 << rng.randint(lo, hi)


def _spread(rng, lo, hi):
    """A whole number spread over the logarithm of [lo, hi]."""
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["build", "lights", "grid", "lookup", "multi", "frame", "pcf", "raster"])
    if kind == "build":
        return {"kind": kind, "n": _log2(rng, 7, 13), "boxes": _spread(rng, 10, 600), "spheres": rng.randint(0, 64),
                "host": rng.random() < 0.25}
    if kind == "lights":
        lo = rng.randint(7, 9)
        return {"kind": kind, "lights": rng.randint(2, 16), "lo": lo, "hi": rng.randint(lo + 1, 12),
                "points": _spread(rng, 1000, 1 << 20)}
    if kind == "grid":
        length = rng.choice([2, 4, 8])
        return {"kind": kind, "length": length, "n": _log2(rng, 8, {2: 12, 4: 11, 8: 10}[length]),
                "points": _spread(rng, 1000, 1 << 22)}
    if kind == "lookup":
        return {"kind": kind, "n": _log2(rng, 7, 13), "points": _spread(rng, 500, 1 << 25), "voxel": rng.random() < 0.3}
    if kind == "multi":
        lo = rng.randint(7, 9)
        return {"kind": kind, "lights": rng.randint(2, 16), "lo": lo, "hi": rng.randint(lo + 1, 12),
                "points": _spread(rng, 1000, 1 << 23)}
    if kind == "frame":
        return {"kind": kind, "n": _log2(rng, 9, 13), "width": rng.randint(320, 3840), "height": rng.randint(240, 2160)}
    if kind == "pcf":
        return {"kind": kind, "n": _log2(rng, 9, 12), "width": rng.randint(320, 1920), "height": rng.randint(240, 1080),
                "filter": rng.choice([2, 3, 4, 5])}
    n = _log2(rng, 8, 12)
    return {"kind": kind, "cells": _spread(rng, 16, 512), "n": n, "width": rng.randint(n // 2, n),
            "height": rng.randint(n // 2, n)}


# ---------------------------------------------------------------- inputs
def _rng(seed, stream=0):
    return np.random.Generator(np.random.PCG64([int(seed), stream]))


def _gen(seed, stream=0):
    return torch.Generator(DEV).manual_seed((int(seed) * 1000003 + stream) & 0x7FFFFFFF)


def _map(n, boxes, spheres, g, plane=0.95):
    """An (n, n) float32 depth map of a plane with boxes and spheres on it."""
    d = torch.full((n, n), plane, dtype=torch.float32, device=DEV)

    def window(c, h):
        return max(0, math.ceil((c - h) * n - 0.5)), min(n, math.floor((c + h) * n - 0.5) + 1)

    c = g.random((boxes, 2))
    h = g.uniform(0.01, 0.08, (boxes, 2))
    top = g.uniform(0.2, 0.85, boxes)
    for k in range(boxes):
        x0, x1 = window(c[k, 0], h[k, 0])
        y0, y1 = window(c[k, 1], h[k, 1])
        if x0 < x1 and y0 < y1:
            d[y0:y1, x0:x1].clamp_(max=float(top[k]))
    c = g.random((spheres, 2))
    r = g.uniform(0.005, 0.05, spheres)
    top = g.uniform(0.2, 0.85, spheres)
    for k in range(spheres):
        x0, x1 = window(c[k, 0], r[k])
        y0, y1 = window(c[k, 1], r[k])
        if x0 < x1 and y0 < y1:
            dx = (torch.arange(x0, x1, device=DEV) + 0.5) / n - c[k, 0]
            dy = (torch.arange(y0, y1, device=DEV) + 0.5) / n - c[k, 1]
            rest = r[k] ** 2 - (dy[:, None] ** 2 + dx[None, :] ** 2)
            z = torch.where(rest > 0, float(top[k]) - rest.clamp_min(0).sqrt(), 2.0)
            d[y0:y1, x0:x1] = torch.minimum(d[y0:y1, x0:x1], z.float())
    return d


def _light_maps(case, seed):
    """One map per light, its side and its scene's box count spread evenly
    over the case's range (sides 2^lo .. 2^hi, 10 .. 2000 boxes)."""
    g, sides = _rng(seed), case["hi"] - case["lo"] + 1
    return [_map(1 << (case["lo"] + i * 5 % sides), int(10 * 200 ** (i * 7 % 16 / 15)), 0, g)
            for i in range(case["lights"])]


def _surface_points(depth, count, gen, out):
    """`count` NDC points into `out`: pixel centres of `depth`, z on the
    surface up to half a voxel off (voxel v at 2 v / (n - 1) - 1)."""
    n = depth.shape[0]
    px = torch.randint(n, (count,), device=DEV, generator=gen)
    py = torch.randint(n, (count,), device=DEV, generator=gen)
    scale = 2.0 / (n - 1)
    out[:, 0] = (px + 0.5) * scale - 1.0
    out[:, 1] = (py + 0.5) * scale - 1.0
    jitter = torch.rand(count, device=DEV, generator=gen) - 0.5
    out[:, 2] = (depth[py, px].double() * n + jitter) * scale - 1.0


def _points(depth, count, gen):
    """Half on the surface, half anywhere in the volume."""
    out = torch.empty((count, 3), dtype=torch.float32, device=DEV)
    half = count // 2
    _surface_points(depth, half, gen, out[:half])
    out[half:] = torch.rand((count - half, 3), device=DEV, generator=gen) * 2 - 1
    return out


def _view(case, depth, seed):
    """The G-buffer of a camera over the scene: neighbouring pixels see
    neighbouring points.  World = (NDC - shift) / extent, so that the light's
    matrix is a scaling and a shift (an orthographic light).  Returns
    positions, normals, albedo (height, width, 4) and the light's matrix."""
    w, h, n = case["width"], case["height"], depth.shape[0]
    g, gen = _rng(seed, 1), _gen(seed, 1)
    # a camera that looks along +v: rows further up see further away
    s = torch.linspace(0, 1, h, device=DEV, dtype=torch.float64)[:, None]
    t = torch.linspace(-0.5, 0.5, w, device=DEV, dtype=torch.float64)[None, :]
    far = 0.25 / (1.25 - s)
    a = g.uniform(0, 2 * math.pi)
    fwd, side = far * 0.8 - 0.4, t * (0.2 + far * 0.5)
    u = (0.5 + math.cos(a) * fwd - math.sin(a) * side).clamp(0.001, 0.999)
    v = (0.5 + math.sin(a) * fwd + math.cos(a) * side).clamp(0.001, 0.999)
    px, py = (u * n).long(), (v * n).long()
    jitter = torch.rand((h, w), device=DEV, generator=gen, dtype=torch.float64) - 0.5
    z = depth[py, px].double() + jitter / n
    ndc = torch.stack([u * 2 - 1, v * 2 - 1, z * 2 - 1], -1)
    extent, shift = g.uniform(0.01, 0.05, 3), g.uniform(-0.1, 0.1, 3)
    pos = torch.ones((h, w, 4), device=DEV)
    pos[..., :3] = (ndc - torch.tensor(shift, device=DEV)) / torch.tensor(extent, device=DEV)
    M = np.eye(4, dtype=np.float32)
    M[:3, :3] = np.diag(extent)
    M[:3, 3] = shift
    nrm = torch.randn((h, w, 4), device=DEV, generator=gen)
    nrm[..., 2] -= 2.0
    nrm /= nrm[..., :3].norm(dim=-1, keepdim=True)
    alb = torch.rand((h, w, 4), device=DEV, generator=gen)
    return pos, nrm, alb, M


LIGHT = (0.3, 0.4, -1.0)


def _terrain(case, seed):
    """Vertex coordinates (cells + 1) and heights of a terrain mesh."""
    cells = case["cells"]
    hgt = 0.3 + 0.5 * torch.rand((cells + 1, cells + 1), device=DEV, generator=_gen(seed))
    return torch.linspace(0, 1, cells + 1, device=DEV), hgt


def _window(case):
    """The rendered window's origin: the map's centre region."""
    return (case["n"] - case["width"]) // 2, (case["n"] - case["height"]) // 2


def _container(depth):
    grid = cp.CompressedShadowContainer.of(cp.CompressedShadow.from_depth(depth))
    grid.move_to_gpu()
    return grid


def _shadows(maps):
    hs = cp.MinMaxHierarchy.create_batch(maps, borrow=True)
    return cp.CompressedShadow.create_batch(hs, [(i, 0, 1) for i in range(len(hs))])


def prepare(case, seed):
    k = case["kind"]
    if k == "build":
        d = _map(case["n"], case["boxes"], case["spheres"], _rng(seed))
        room = case["n"] ** 2 // 4 + (1 << 18)  # several times any such scene's DAG
        if not case["host"]:
            return {"case": case, "depth": d, "words": torch.zeros(room, dtype=torch.int32, device=DEV)}
        host = torch.empty(d.shape, dtype=torch.float32, pin_memory=True)
        host.copy_(d)
        words = torch.empty(room, dtype=torch.int32, pin_memory=True).zero_()
        return {"case": case, "depth": host, "words": words}
    if k in ("lights", "multi"):
        maps = _light_maps(case, seed)
        gen = _gen(seed)
        ids = torch.randint(len(maps), (case["points"],), device=DEV, generator=gen, dtype=torch.int32)
        pts = torch.rand((case["points"], 3), device=DEV, generator=gen) * 2 - 1
        for i, d in enumerate(maps):  # half of each light's points on its surface
            mine = torch.nonzero(ids == i)[::2, 0]
            near = torch.empty((mine.numel(), 3), device=DEV)
            _surface_points(d, mine.numel(), gen, near)
            pts[mine] = near
        s = {"case": case, "ids": ids, "points": pts,
             "out": torch.empty((case["points"] + 31) // 32, dtype=torch.int32, device=DEV)}
        return {**s, "maps": maps} if k == "lights" else {**s, "shadows": _shadows(maps)}
    if k == "grid":
        L, n = case["length"], case["n"]
        d = _map(L * n, 100 * L, 16 * L, _rng(seed))
        tiles = [d[y * n:(y + 1) * n, x * n:(x + 1) * n].contiguous() for y in range(L) for x in range(L)]
        return {"case": case, "tiles": tiles, "points": _points(d, case["points"], _gen(seed))}
    if k == "lookup":
        d = _map(case["n"], min(500, case["n"] // 16 + 8), case["n"] // 128, _rng(seed))
        pts = _points(d, case["points"], _gen(seed))
        if case["voxel"]:
            pts = ((pts + 1) * 0.5 * (case["n"] - 1)).int()
        out = torch.empty((case["points"] + 31) // 32, dtype=torch.int32, device=DEV)
        return {"case": case, "shadow": cp.CompressedShadow.from_depth(d), "points": pts, "out": out}
    if k in ("frame", "pcf"):
        d = _map(case["n"], 500, 64, _rng(seed))
        pos, nrm, alb, M = _view(case, d, seed)
        grid = _container(d)
        if k == "pcf":
            grid.set_filter_size(case["filter"])
        s = {"case": case, "grid": grid, "pos": pos, "M": M,
             "vis": torch.empty(pos.shape[:2], dtype=torch.uint8, device=DEV)}
        return s if k == "pcf" else {**s, "nrm": nrm, "alb": alb, "rgba": torch.empty_like(alb)}
    c, hgt = _terrain(case, seed)
    X, Y = c[None, :].expand_as(hgt), c[:, None].expand_as(hgt)
    v = torch.stack([X, Y, hgt], -1)
    a, b, d, e = v[:-1, :-1], v[:-1, 1:], v[1:, :-1], v[1:, 1:]
    tris = torch.stack([torch.cat([a, b, e], -1), torch.cat([a, e, d], -1)], 2).reshape(-1, 9).contiguous()
    return {"case": case, "tris": tris}


class _Dag:
    """The device words of a resident shadow, for torch, which keeps this
    object (and so the shadow) while it uses them."""

    def __init__(self, shadow):
        self.shadow = shadow
        self.__cuda_array_interface__ = {"shape": (shadow.dag_size(),), "typestr": "<i4", "version": 2,
                                         "data": (shadow.device_dag(), False)}


def run(s):
    case = s["case"]
    k = case["kind"]
    if k == "build":
        sh = cp.CompressedShadow.from_depth(s["depth"])
        if case["host"]:
            sh.get_dag(out=s["words"])
        else:
            s["words"][:sh.dag_size()].copy_(torch.as_tensor(_Dag(sh), device=DEV))
        return s["words"], sh.dag_size(), sh.get_total_visibility()
    if k == "grid":
        grid = cp.CompressedShadowContainer(case["length"])
        grid.build(cp.MinMaxHierarchy.create_batch(s["tiles"], borrow=True))
        return grid.lookup_ndc(s["points"])
    if k == "lookup":
        sh = s["shadow"]
        return (sh.lookup_voxel if case["voxel"] else sh.lookup_ndc)(s["points"], out=s["out"])
    if k in ("lights", "multi"):
        return cp.lookup_ndc_multi(_shadows(s["maps"]) if k == "lights" else s["shadows"],
                                   s["ids"], s["points"], out=s["out"])
    if k == "pcf":
        return s["grid"].evaluate(s["pos"], s["M"], out=s["vis"])
    if k == "frame":
        vis = s["grid"].evaluate(s["pos"], s["M"], out=s["vis"])
        rgba = cp.shade(s["nrm"], s["alb"], LIGHT, visibilities=vis, out=s["rgba"], stream=torch.cuda.current_stream())
        return vis, rgba
    x0, y0 = _window(case)
    return cp.raster_triangles(s["tris"], case["n"], 1.0, x0, y0, case["width"], case["height"])


def work(case):
    """Bytes of inputs read once and outputs written once (DAG words counted
    at 0.036 of the map's bytes, as the benchmark's scenes give them)."""
    k = case["kind"]
    if k == "build":
        b = 4 * case["n"] ** 2
        return {"bytes": b * 1.036, "flops": 0}
    if k == "lights":
        sides = case["hi"] - case["lo"] + 1
        b = sum(4 * (1 << (case["lo"] + i * 5 % sides)) ** 2 for i in range(case["lights"]))
        return {"bytes": b + case["points"] * 16.125, "flops": 0}
    if k == "grid":
        return {"bytes": 4 * (case["length"] * case["n"]) ** 2 + case["points"] * 12.125, "flops": 0}
    if k == "lookup":
        return {"bytes": case["points"] * 12.125, "flops": 0}
    if k == "multi":
        return {"bytes": case["points"] * 16.125, "flops": 0}
    if k in ("frame", "pcf"):
        return {"bytes": case["width"] * case["height"] * (65 if k == "frame" else 17), "flops": 0}
    # the window's share of the mesh, and the window
    share = case["width"] * case["height"] / case["n"] ** 2
    return {"bytes": 72 * case["cells"] ** 2 * share + 4 * case["width"] * case["height"], "flops": 0}


def exact(case, seed):
    """The floating-point outputs in 64 bits; DAG words, bits and visibility
    bytes are whole numbers and have none."""
    if case["kind"] == "frame":
        d = _map(case["n"], 500, 64, _rng(seed))
        pos, nrm, alb, M = _view(case, d, seed)
        n = case["n"]
        ndc = pos[..., :3].double() * torch.tensor(M[:3, :3].diagonal().copy(), device=DEV).double() + \
            torch.tensor(M[:3, 3], device=DEV).double()
        q = ((ndc + 1) * 0.5 * (n - 1)).trunc().long()  # the voxel, lit when its centre is above the surface
        lit = (q[..., 2] + 0.5 <= d[q[..., 1].clamp(0, n - 1), q[..., 0].clamp(0, n - 1)].double() * n).double()
        light = torch.tensor(LIGHT, device=DEV).double()
        dot = (nrm[..., :3].double() * (light / light.norm())).sum(-1).clamp_min(0)
        rgba = alb.double()
        rgba[..., :3] *= (0.15 + dot * lit)[..., None]
        return None, rgba
    if case["kind"] != "raster":
        return None
    c, hgt = _terrain(case, seed)
    c, hgt, cells, n = c.double(), hgt.double(), case["cells"], case["n"]
    x0, y0 = _window(case)

    def axis(o, size):  # cell of each pixel centre, and the place in it
        p = (torch.arange(o, o + size, device=DEV).double() + 0.5) / n
        i = (torch.searchsorted(c, p, right=True) - 1).clamp(0, cells - 1)
        return i, (p - c[i]) / (c[i + 1] - c[i])

    (i, u), (j, v) = axis(x0, case["width"]), axis(y0, case["height"])
    i, u, j, v = i[None, :], u[None, :], j[:, None], v[:, None]
    a, b, d, e = hgt[j, i], hgt[j, i + 1], hgt[j + 1, i], hgt[j + 1, i + 1]
    return torch.where(u >= v, a + u * (b - a) + v * (e - b), a + v * (d - a) + u * (e - d))
