"""Kernels whose start overlaps the end of the kernel before them (csrc/launch.cuh): the sources, where what that
kernel writes must not be read as if it were read-only for the kernel's lifetime (a race that a correct run does not
show), and builds and small renders issued back to back, with changing inputs and on two streams."""
import os
import re

import numpy as np
import pytest

import gr
from gr import scenes as sc

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "gpu-renderer_gb300", "csrc")
# read-only while these grids exist: their writer has ended when the build's first kernel lets them start
READ_ONLY = {("k_morton_hist", "verts"), ("k_climb_chunk", "verts")}


def _block(text, at, opening, closing):
    """The text from the first `opening` at or after `at` to its `closing`."""
    i = text.index(opening, at)
    depth = 0
    for j in range(i, len(text)):
        depth += (text[j] == opening) - (text[j] == closing)
        if depth == 0:
            return i, j + 1
    raise AssertionError("unbalanced")


def _kernels(source):
    """Name, parameters and body of every kernel that `source` launches overlapped."""
    text = re.sub(r"//[^\n]*", "", open(os.path.join(CSRC, source)).read())
    names = set(re.findall(r"launch_after\(\s*\w+,\s*(k_\w+)", text))
    assert names
    for name in sorted(names):
        at = next(m.start() for m in re.finditer(r"\b%s\s*\(" % name, text)
                  if "__global__" in text[max(0, m.start() - 120):m.start()])
        p0, p1 = _block(text, at, "(", ")")
        b0, b1 = _block(text, p1, "{", "}")
        yield name, text[p0 + 1:p1 - 1], text[b0:b1], text


@pytest.mark.parametrize("source", ["lbvh.cu", "render.cu"])
def test_overlapped_kernels_wait_and_read_coherently(source):
    for name, params, body, text in _kernels(source):
        assert "wait_for_previous();" in body, name
        for p in params.split(","):
            if "__restrict__" in p:
                assert "const" in p and (name, p.split()[-1]) in READ_ONLY, (name, p.strip())
        for arg in re.findall(r"__ldg\(([^()]*)", body):
            assert arg == "v + k" and (name, "verts") in READ_ONLY, (name, arg)  # a triangle's vertices
        if "tri_box" in body:
            assert ("tri_box<true>" in body) == ((name, "verts") in READ_ONLY), name
    # what a wave's traversal reads through its source of rays
    if source == "render.cu":
        i, j = _block(text, text.index("struct WaveSrc"), "{", "}")
        assert "__ldg" not in text[i:j] and "__restrict__" not in text[i:j]


@pytest.mark.gpu
@pytest.mark.parametrize("n", [300, 3001, 100003])
def test_builds_back_to_back(ctx, oracle, n):
    """Vertices written by the kernel just before each build, no wait in between; then two BVHs on two streams in turn."""
    import torch
    soups = [sc.triangle_soup(n, seed_salt=900 + k) for k in range(6)]
    want = [oracle.lbvh(v) for v in soups]
    dev = [torch.from_numpy(v.reshape(n, 9)).cuda() for v in soups]
    verts = [torch.empty(n, 9, dtype=torch.float32, device="cuda") for _ in range(2)]
    bvhs = [gr.BVH(ctx) for _ in range(2)]
    streams = [torch.cuda.Stream(), torch.cuda.Stream()]
    torch.cuda.synchronize()

    def check(b, w):
        got = b.export()
        for k in ("root", "sorted_prim", "sorted_code", "nodes"):
            np.testing.assert_array_equal(got[k], w[k], err_msg=k)

    for k in range(6):  # one stream, one BVH after the other
        with torch.cuda.stream(streams[0]):
            torch.mul(dev[k], 1.0, out=verts[0])
            bvhs[0].build_device(verts[0], n, stream=streams[0].cuda_stream)
            if k:  # the next vertices are written while nothing has been waited for
                torch.mul(dev[k - 1], 1.0, out=verts[0])
                bvhs[1].build_device(verts[0], n, stream=streams[0].cuda_stream)
        streams[0].synchronize()
        check(bvhs[0], want[k])
        if k:
            check(bvhs[1], want[k - 1])
    for k in range(0, 6, 2):
        for s, b, v, j in zip(streams, bvhs, verts, (k, k + 1)):
            with torch.cuda.stream(s):
                torch.mul(dev[j], 1.0, out=v)
                b.build_device(v, n, stream=s.cuda_stream)
        for s in streams:
            s.synchronize()
        check(bvhs[0], want[k])
        check(bvhs[1], want[k + 1])
    for b in bvhs:
        b.close()


@pytest.mark.gpu
@pytest.mark.parametrize("layout", [gr.LAYOUT_BVH2, gr.LAYOUT_BVH8_Q8])
def test_small_waves_back_to_back(ctx, layout):
    """A render in many small waves, whose kernels follow each other without a wait, against the same in one wave and with
    launches in place of a graph; two scenes in turn."""
    scenes = [gr.Scene(ctx, d) for d in (sc.textured_scene(61, 37), sc.cornell_box(40, 31))]
    got = []
    for wave_paths, flags in ((0, 0), (1, 0), (1, gr.RENDER_NO_GRAPH)):
        for s in scenes:
            s.set_tuning(layout, 64, 12)
            s.reset()
        for k in range(2):
            for s in scenes:
                s.render(7, max_depth=6, seed=21 + k, wave_paths=wave_paths, flags=flags)
        got.append([s.accumulation()[0] for s in scenes])
    for other in got[1:]:
        for a, b in zip(got[0], other):
            np.testing.assert_array_equal(a, b)
    for s in scenes:
        s.close()


@pytest.mark.gpu
@pytest.mark.parametrize("replay", [False, True])
def test_a_captured_first_build_leaves_the_next_one_sound(ctx, oracle, replay):
    """The first build of a BVH, which allocates, recorded into a graph; the next one runs at once, whether the graph has been
    launched or not. The memory that the BVH gets held other values before."""
    import torch
    n = 3001
    v, w = sc.triangle_soup(n, seed_salt=920), sc.triangle_soup(n, seed_salt=921)
    dv, dw = (torch.from_numpy(x.reshape(n, 9)).cuda() for x in (v, w))
    for size in (1 << 12, 1 << 16, 1 << 18, 1 << 20, 1 << 26):
        dirty = [torch.full((size,), 255, dtype=torch.uint8, device="cuda") for _ in range(4)]
        torch.cuda.synchronize()
        del dirty
    torch.cuda.empty_cache()
    b, st, g = gr.BVH(ctx), torch.cuda.Stream(), torch.cuda.CUDAGraph()
    warm = gr.BVH(ctx)
    warm.build_device(dv, n)  # kernels loaded
    torch.cuda.synchronize()
    with torch.cuda.graph(g, stream=st, capture_error_mode="relaxed"):
        b.build_device(dv, n, stream=torch.cuda.current_stream().cuda_stream)
    steps = [lambda: b.build_device(dw, n, stream=st.cuda_stream)]
    want = [oracle.lbvh(w)]
    if replay:
        steps = [g.replay] + steps + [g.replay]
        want = [oracle.lbvh(v)] + want + [oracle.lbvh(v)]
    for step, tree in zip(steps, want):
        with torch.cuda.stream(st):
            step()
        st.synchronize()
        got = b.export()
        for k in ("root", "sorted_prim", "sorted_code", "nodes"):
            np.testing.assert_array_equal(got[k], tree[k], err_msg=k)
    warm.close()
    b.close()
