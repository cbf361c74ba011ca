"""Performance cases: the work that programs built on gr have it do, through its public entry points.

Five kinds of work, each over the range of sizes that it meets:

  trace   rays already on the GPU against a resident BVH (gr_trace): closest hit or any hit, from a picking query of a
          few hundred rays to millions; binary nodes (the default) or the 8-wide nodes the autotuner picks
  host    the same with rays and hits in host memory (gr_trace_host), pageable as numpy gives it or page-locked
  tree    an LBVH built into the caller's own buffers (gr_bvh_build_noalloc), which come back whole
  frame   geometry that moves: the BVH is rebuilt from new vertices and rays are traced against it (gr_bvh_build + gr_trace)
  render  a scene rendered from scratch (gr_scene_reset + gr_render), the image to the host or to the GPU
  batch   several scenes in shared waves (gr_render_batch), then their images' sums

The soups, rays and scenes are those of gr.scenes (triangle centroids uniform in the unit cube, lognormal edge lengths, scaled
with the number of triangles so that a soup keeps its density; Cornell box, textured scene, displaced spheres).
"""
import ctypes
import math
import os
import sys

import numpy as np
import torch

_ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
_PKG = os.path.join(_ROOT, "gpu-renderer_gb300")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

import gr  # noqa: E402
from gr import scenes  # noqa: E402

# Rays leave the unit cube before this distance: a miss keeps it as its t.
FAR = 4.0
TREE_LIMIT = 131072  # gr_bvh_build_noalloc's

_P = ctypes.c_void_p
_ctx = None


def context():
    """The program's one context."""
    global _ctx
    if _ctx is None:
        _ctx = gr.Context(0)
    return _ctx


def listed():
    return [
        # a pick or a collision query: a handful of rays, the default configuration; launch and latency
        {"name": "pick_1k", "kind": "trace", "tris": 20011, "rays": 1021, "query": "incoherent", "layout": gr.LAYOUT_BVH2},
        # the traversal microbenchmark's size (bench.py's headline): diffuse bounces in a million triangles
        {"name": "closest_4m", "kind": "trace", "tris": 1000000, "rays": 4194304, "query": "incoherent",
         "layout": gr.LAYOUT_BVH8_Q8},
        # a lighting or visibility pass: any hit between pairs of points
        {"name": "shadow_1m", "kind": "trace", "tris": 262147, "rays": 1000003, "query": "shadow",
         "layout": gr.LAYOUT_BVH8_Q8},
        # a viewer's primary rays with the default configuration, 1024 x 768
        {"name": "camera_default", "kind": "trace", "tris": 300007, "rays": 786432, "query": "camera",
         "layout": gr.LAYOUT_BVH2},
        # rays in numpy arrays, as a script has them
        {"name": "host_400k", "kind": "host", "tris": 100003, "rays": 400009, "query": "incoherent",
         "layout": gr.LAYOUT_BVH8_Q8, "pinned": False},
        # a plug-in's per-call build into its host application's buffers
        {"name": "tree_100k", "kind": "tree", "tris": 100003},
        # a small moving mesh, rebuilt and queried every frame
        {"name": "frame_3k", "kind": "frame", "tris": 3001, "rays": 2048, "query": "incoherent", "layout": gr.LAYOUT_BVH2},
        # a large moving mesh rebuilt every frame into the autotuned layout
        {"name": "frame_1m", "kind": "frame", "tris": 1000000, "rays": 262144, "query": "incoherent",
         "layout": gr.LAYOUT_BVH8_Q8},
        # a thumbnail or an interactive preview frame while the camera moves
        {"name": "preview", "kind": "render", "scene": "textured", "level": 0, "width": 160, "height": 120, "spp": 1,
         "depth": 8, "layout": gr.LAYOUT_BVH2, "host": True},
        # the Cornell-box configuration: 256 x 256, 16 spp, depth 8
        {"name": "cornell_256", "kind": "render", "scene": "cornell", "level": 0, "width": 256, "height": 256, "spp": 16,
         "depth": 8, "layout": gr.LAYOUT_BVH8_Q8, "host": True},
        # the glossy configuration: 5.26M triangles, 1024 x 768, 64 spp, depth 16, the image left on the GPU
        {"name": "glossy_1024", "kind": "render", "scene": "glossy", "level": 8, "width": 1024, "height": 768, "spp": 64,
         "depth": 16, "layout": gr.LAYOUT_BVH8_Q8, "host": False},
        # a queue of small render jobs in shared waves
        {"name": "batch_8", "kind": "batch", "jobs": 8, "max_tris": 200000, "res": 200, "spp": 8, "depth": 8,
         "layout": gr.LAYOUT_BVH8_Q8},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["trace", "trace", "host", "tree", "frame", "frame", "render", "render", "batch"])
    layout = rng.choice([gr.LAYOUT_BVH2, gr.LAYOUT_BVH8_Q8, gr.LAYOUT_BVH8_Q8])
    query = rng.choice(["incoherent", "shadow", "camera"])
    if kind == "trace":
        return {"kind": kind, "tris": _log(rng, 500, 1000000), "rays": _log(rng, 256, 4194304), "query": query,
                "layout": layout}
    if kind == "host":
        return {"kind": kind, "tris": _log(rng, 500, 1000000), "rays": _log(rng, 256, 2000000), "query": query,
                "layout": layout, "pinned": rng.random() < 0.5}
    if kind == "tree":
        return {"kind": kind, "tris": _log(rng, 32, TREE_LIMIT)}
    if kind == "frame":
        return {"kind": kind, "tris": _log(rng, 32, 3000000), "rays": _log(rng, 256, 262144), "query": query,
                "layout": layout}
    if kind == "render":
        scene = rng.choice(["textured", "cornell", "glossy"])
        width, height = _log(rng, 96, 1024), _log(rng, 72, 768)
        return {"kind": kind, "scene": scene, "level": rng.randint(3, 7) if scene == "glossy" else 0, "width": width,
                "height": height, "spp": _log(rng, 1, 64), "depth": rng.randint(4, 16), "layout": layout,
                "host": rng.random() < 0.7}
    return {"kind": kind, "jobs": rng.randint(2, 12), "max_tris": _log(rng, 20000, 200000), "res": _log(rng, 100, 300),
            "spp": rng.randint(2, 16), "depth": rng.randint(4, 12), "layout": layout}


# ---- inputs ------------------------------------------------------------------------


def _generator(seed, salt):
    return torch.Generator(device="cuda").manual_seed((int(seed) * 1000003 + salt) & 0x7FFFFFFF)


def _unit(g, n):
    d = torch.randn(n, 3, generator=g, device="cuda", dtype=torch.float64)
    return d / d.norm(dim=1, keepdim=True)


def _soup(n, seed, salt=1):
    """gr.scenes.triangle_soup on the GPU, edges scaled to keep its 1M-triangle density at other sizes."""
    g = _generator(seed, salt)
    c = torch.rand(n, 1, 3, generator=g, device="cuda", dtype=torch.float64)
    size = math.exp(-6.0) * (1.0e6 / n) ** 0.5
    s = torch.exp(0.5 * torch.randn(n, 3, 1, generator=g, device="cuda", dtype=torch.float64)) * min(size, 0.2)
    v = c + s * _unit(g, 3 * n).view(n, 3, 3)
    return v.to(torch.float32).reshape(n, 9).contiguous()


def _rays(n, query, seed):
    g = _generator(seed, 2)
    r = torch.empty(n, 8, dtype=torch.float32, device="cuda")
    r[:, 6] = 0.0
    if query == "camera":  # pixel-centre pinhole rays over a grid of about 4 : 3, row by row, from a seeded eye
        w = max(1, int(math.sqrt(n * 4.0 / 3.0)))
        eye = torch.tensor([0.5, 0.5, -1.0], dtype=torch.float64, device="cuda")
        eye = eye + 0.1 * torch.rand(3, generator=g, device="cuda", dtype=torch.float64)
        i = torch.arange(n, device="cuda")
        x = ((i % w).double() + 0.5) / w * 2.0 - 1.0
        y = 1.0 - ((i // w).double() + 0.5) / max(1.0, n / w) * 2.0
        t = math.tan(math.radians(40.0) * 0.5)
        d = torch.stack([x * t, y * t * 0.75, torch.ones_like(x)], dim=1)
        r[:, 0:3] = eye.float()
        r[:, 3:6] = (d / d.norm(dim=1, keepdim=True)).float()
        r[:, 7] = FAR
    else:
        r[:, 0:3] = torch.rand(n, 3, generator=g, device="cuda")
        if query == "shadow":  # to a second point, d not normalised (the renderer's shadow rays)
            r[:, 3:6] = torch.rand(n, 3, generator=g, device="cuda") - r[:, 0:3]
            r[:, 7] = 0.9999
        else:
            r[:, 3:6] = _unit(g, n).float()
            r[:, 7] = FAR
    return r


def _displaced(level, radius, center, r):
    """A sphere displaced by a few seeded sine waves (amplitude 0.05), with its smooth normals."""
    V, F = scenes.icosphere(level)
    disp, grad = np.ones(V.shape[0]), np.zeros_like(V)
    for _ in range(5):
        f, p = r.normal(0.0, 4.0, 3), r.uniform(0.0, 2.0 * np.pi)
        a = V @ f + p
        disp += 0.02 * np.sin(a)
        grad += 0.02 * np.cos(a)[:, None] * f
    N = V * disp[:, None] - (grad - np.sum(grad * V, axis=1, keepdims=True) * V)
    N /= np.linalg.norm(N, axis=1, keepdims=True)
    P = V * disp[:, None] * radius + np.asarray(center)
    return P.astype(np.float32), F.astype(np.uint32), N.astype(np.float32)


def _glossy(width, height, level, seed):
    """The glossy configuration's scene (gr.scenes.glossy_scene) with spheres displaced from the seed."""
    d = scenes.glossy_scene(width, height, level=2, glass_level=max(0, level - 3))
    r = np.random.default_rng(int(seed))
    for i, x in enumerate((-1.65, -0.55, 0.55, 1.65)):
        P, F, N = _displaced(level, 0.5, (x, 0.55, 0.0), r)
        d.meshes[2 + i] = scenes.MeshDesc(P, F, 3 + i, normals=N)
    return d


def _scene(case, seed):
    if case["scene"] == "glossy":
        return _glossy(case["width"], case["height"], case["level"], seed)
    make = scenes.cornell_box if case["scene"] == "cornell" else scenes.textured_scene
    return make(case["width"], case["height"], seed_salt=int(seed) % 100000)


def _tune(thing, layout):
    """The default configuration, or for 8-wide nodes the launch shape the autotuner picks."""
    if layout == gr.LAYOUT_BVH8_Q8:
        thing.set_tuning(layout, 64, 12)
    else:
        thing.set_tuning(layout)


def prepare(case, seed):
    ctx, kind = context(), case["kind"]
    if kind in ("trace", "host", "frame"):
        s = {"bvh": gr.BVH(ctx), "verts": _soup(case["tris"], seed), "rays": _rays(case["rays"], case["query"], seed)}
        s["any"] = case["query"] == "shadow"
        torch.cuda.synchronize()
        if kind == "frame":  # the frame before: other vertices
            s["bvh"].build_device(_soup(case["tris"], seed, salt=3), case["tris"])
        else:
            s["bvh"].build_device(s["verts"], case["tris"])
        torch.cuda.synchronize()
        _tune(s["bvh"], case["layout"])
        if kind == "host":
            rays = s.pop("rays")
            if case["pinned"]:
                s["rays"] = rays.cpu().pin_memory()
                s["hits"] = torch.zeros(case["rays"], 4, dtype=torch.float32).pin_memory()
            else:
                s["rays"] = rays.cpu().numpy()
        else:
            s["hits"] = torch.zeros(case["rays"], 4, dtype=torch.float32, device="cuda")
    elif kind == "tree":
        n = case["tris"]
        new = lambda words, t=torch.int32: torch.zeros(words, dtype=t, device="cuda")  # noqa: E731
        s = {"verts": _soup(n, seed), "nodes": new(16 * max(n - 1, 1)), "tris": new(12 * n, torch.float32), "prim": new(n),
             "code": new(n), "header": new(16)}
        f = gr.load().gr_bvh_build_noalloc
        f.argtypes, f.restype = [_P, _P, ctypes.c_uint32, _P, _P, _P, _P, _P, _P], ctypes.c_int
    elif kind == "render":
        s = {"scene": gr.Scene(ctx, _scene(case, seed)), "seed": int(seed) + 1, "out": None}
        _tune(s["scene"], case["layout"])
        if not case["host"]:
            s["out"] = torch.zeros(case["height"], case["width"], 3, dtype=torch.float32, device="cuda")
    else:
        s = {"scenes": [], "opts": []}
        for j in range(case["jobs"]):
            desc, _ = scenes.batch_job(int(seed) * 16 + j, max_tris=case["max_tris"])
            side = case["res"] * (1, 2, 4)[j % 3] // 2
            desc.camera["width"], desc.camera["height"] = side + j, side
            s["scenes"].append(gr.Scene(ctx, desc))
            _tune(s["scenes"][-1], case["layout"])
            s["opts"].append({"spp": case["spp"] * (1 + j % 4), "max_depth": case["depth"], "seed": int(seed) + j})
    s["case"] = case
    torch.cuda.synchronize()
    return s


# ---- one pass ----------------------------------------------------------------------


def _hits(t, i):
    """A hit record's fields: t and the barycentrics as floats, the triangle as an integer."""
    return {"t": t[:, 0], "prim": i[:, 1], "uv": t[:, 2:4]}


def run(s):
    case = s["case"]
    kind, ctx = case["kind"], context()
    if kind == "trace" or kind == "frame":
        if kind == "frame":
            s["bvh"].build_device(s["verts"], case["tris"])
        s["bvh"].trace_device(s["rays"], case["rays"], s["hits"], any_hit=s["any"])
        return _hits(s["hits"], s["hits"].view(torch.int32))
    if kind == "host":
        if case["pinned"]:
            ctx.check(gr.load().gr_trace_host(s["bvh"].h, s["rays"].data_ptr(), case["rays"], s["hits"].data_ptr(),
                                              int(s["any"])), "gr_trace_host")
            return _hits(s["hits"], s["hits"].view(torch.int32))
        h = s["bvh"].trace_host(s["rays"], any_hit=s["any"])
        return _hits(h, h.view(np.int32))
    if kind == "tree":
        p = [s[k].data_ptr() for k in ("verts", "nodes", "tris", "prim", "code", "header")]
        st = gr.load().gr_bvh_build_noalloc(ctx.h, p[0], case["tris"], *p[1:], torch.cuda.current_stream().cuda_stream)
        ctx.check(st, "gr_bvh_build_noalloc")
        return {k: s[k] for k in ("nodes", "tris", "prim", "code", "header")}
    if kind == "render":
        s["scene"].reset()
        img, st = s["scene"].render(case["spp"], case["depth"], s["seed"], out=s["out"])
        return {"image": img, "closest_rays": int(st.closest_rays), "shadow_rays": int(st.shadow_rays)}
    for sc in s["scenes"]:
        sc.reset()
    st = gr.render_batch(ctx, s["scenes"], s["opts"])
    sums = [sc.accumulation()[0] for sc in s["scenes"]]
    return {"sums": sums, "closest_rays": int(st.closest_rays), "shadow_rays": int(st.shadow_rays)}


# ---- what a pass cannot do without -----------------------------------------------------

RAY, HIT, TRI, NODE, LEAF = 32, 16, 36, 64, 48  # bytes: records of gr.h
BOX, TEST, SHADE = 18, 50, 150                  # operations: a box, a triangle, a shading point


def _query_flops(rays, tris):
    """One path from the root to a leaf, both boxes of each node, and one triangle."""
    return rays * (2 * BOX * max(1.0, math.log2(tris)) + TEST)


def _camera_paths(w, h, spp, depth, tris, image_bytes):
    """Every path's camera ray, and for half of its bounces (up to 4) a scatter ray, a shadow ray and a shading point."""
    paths = w * h * spp
    rays = paths * (1 + 2 * min(4, depth / 2.0))
    return {"bytes": w * h * image_bytes + tris * TRI, "flops": _query_flops(rays, tris) + 0.5 * rays * SHADE}


def work(case):
    kind = case["kind"]
    if kind in ("trace", "host", "frame"):
        n, m = case["tris"], case["rays"]
        b = n * TRI + m * (RAY + HIT)
        if kind == "frame":
            b += n * (NODE + LEAF)
        return {"bytes": b, "flops": _query_flops(m, n)}
    if kind == "tree":
        return {"bytes": case["tris"] * (TRI + NODE + LEAF + 8), "flops": case["tris"] * 60}
    if kind == "render":
        tris = 4 * 20 * 4 ** case["level"] if case["scene"] == "glossy" else 700
        return _camera_paths(case["width"], case["height"], case["spp"], case["depth"], tris, 12)
    total = {"bytes": 0.0, "flops": 0.0}
    for j in range(case["jobs"]):
        side = case["res"] * (1, 2, 4)[j % 3] // 2
        w = _camera_paths(side + j, side, case["spp"] * (1 + j % 4), case["depth"], case["max_tris"] / 3, 24)
        total = {k: total[k] + w[k] for k in total}
    return total


# ---- in 64 bits --------------------------------------------------------------------


def exact(case, seed):
    """Closest hits by testing every ray against every triangle in 64 bits (Moeller-Trumbore), where that takes seconds. Any hit
    may answer with any triangle on the ray; trees are orders and copies of input coordinates; a render's paths are random walks
    that one rounding sends elsewhere."""
    if case["kind"] not in ("trace", "host", "frame") or case["query"] == "shadow" or case["tris"] * case["rays"] > 5e10:
        return None
    tri = _soup(case["tris"], seed).double().view(-1, 3, 3)
    rays = _rays(case["rays"], case["query"], seed).double()
    a, e1, e2 = tri[:, 0], tri[:, 1] - tri[:, 0], tri[:, 2] - tri[:, 0]
    n = torch.linalg.cross(e1, e2)
    na = (n * a).sum(1)
    out_t = torch.empty(len(rays), dtype=torch.float64, device="cuda")
    out_uv = torch.zeros(len(rays), 2, dtype=torch.float64, device="cuda")
    # det, and the two barycentrics times it, are bilinear in (d, o x d) and the triangle: three matrix products
    step = max(1, int(2.0e8 // len(tri)))
    for i in range(0, len(rays), step):
        o, d, tmin, tmax = rays[i:i + step, 0:3], rays[i:i + step, 3:6], rays[i:i + step, 6:7], rays[i:i + step, 7:8]
        m = torch.linalg.cross(o, d)
        det = -(d @ n.T)
        u = (m @ e2.T + d @ torch.linalg.cross(a, e2).T) / det
        v = (d @ torch.linalg.cross(e1, a).T - m @ e1.T) / det
        t = (o @ n.T - na) / det
        t = torch.where((u >= 0) & (v >= 0) & (u + v <= 1) & (t >= tmin) & (t <= tmax), t, torch.inf)
        best, k = t.min(dim=1, keepdim=True)
        hit = torch.isfinite(best)
        out_t[i:i + step] = torch.where(hit, best, tmax)[:, 0]
        out_uv[i:i + step] = torch.where(hit, torch.cat([u.gather(1, k), v.gather(1, k)], dim=1), 0.0)
    if case["kind"] == "host":
        out_t, out_uv = out_t.cpu(), out_uv.cpu()
    return {"t": out_t, "prim": None, "uv": out_uv}
