"""Builds that fail report it, and what they leave is not traversed: the 8-wide build after a binary build whose device
wait gave up (its error word, set by hand), and a rebuild whose 8-wide nodes find no memory."""
import numpy as np
import pytest

import gr
from gr import scenes as sc

pytestmark = pytest.mark.gpu
INVALID, OOM, TIMEOUT = 1, 3, 5


def fill_gpu(leave):
    """Tensors that take the GPU's memory but for about `leave` bytes."""
    import torch
    torch.cuda.empty_cache()
    held = []
    size = 1 << 36
    while size >= 1 << 21:
        free = torch.cuda.mem_get_info()[0]
        if free - size < leave:
            size >>= 1
            continue
        try:
            held.append(torch.empty(size, dtype=torch.uint8, device="cuda"))
        except torch.cuda.OutOfMemoryError:
            size >>= 1
    return held


@pytest.mark.parametrize("n", [1, 5, 300, 20011])
def test_error_of_the_binary_build_stops_the_8_wide_build(ctx, oracle, n):
    v = sc.triangle_soup(n, seed_salt=880 + n)
    rays = sc.incoherent_rays(500, seed_salt=881)
    tree = oracle.lbvh(v)
    b = gr.BVH(ctx)
    b.build_host(v)
    ctx.check(gr.load().gr_diag_set_build_error(b.h, 1), "gr_diag_set_build_error")
    for _ in range(2):
        with pytest.raises(gr.GrError) as e:
            b.set_layout(gr.LAYOUT_BVH8_Q8)
        assert e.value.status == TIMEOUT
    assert b.tuning()["layout"] == gr.LAYOUT_NAMES[gr.LAYOUT_BVH2]
    b.build_host(v)  # clears the word
    b.set_layout(gr.LAYOUT_BVH8_Q8)
    np.testing.assert_array_equal(b.export_layout(gr.LAYOUT_BVH8_Q8), oracle.bvh8(tree)[0])
    np.testing.assert_array_equal(b.trace_host(rays).view(np.uint32), oracle.trace(tree, rays).view(np.uint32))
    b.close()


def test_nodes_that_found_no_memory_are_not_traversed(oracle):
    import torch
    ctx = gr.Context(0)  # its own: the 8-wide build's memory must not be grown yet
    n, m = 1000000, 1000
    v = sc.triangle_soup(n, seed_salt=884)
    big = torch.from_numpy(v.reshape(n, 9)).cuda()
    rays = sc.incoherent_rays(m, seed_salt=885)
    d_rays, d_hits = torch.from_numpy(rays).cuda(), torch.zeros(m, 4, dtype=torch.float32, device="cuda")
    b = gr.BVH(ctx)
    b.build_device(big, n)  # the binary build's memory
    b.build_device(big, 1000)
    b.set_layout(gr.LAYOUT_BVH8_Q8)
    torch.cuda.synchronize()
    held = fill_gpu(64 << 20)  # the 8-wide build of a million triangles takes 136 MB
    try:
        with pytest.raises(gr.GrError) as e:
            b.build_device(big, n)
        assert e.value.status == OOM
        with pytest.raises(gr.GrError) as e:
            b.trace_device(d_rays, m, d_hits)
        assert e.value.status == INVALID
        b.set_layout(gr.LAYOUT_BVH2)  # the binary nodes are there
        b.trace_device(d_rays, m, d_hits)
        torch.cuda.synchronize()
    finally:
        del held
        torch.cuda.empty_cache()
    want = oracle.trace(oracle.lbvh(v), rays).view(np.uint32)
    np.testing.assert_array_equal(d_hits.cpu().numpy().view(np.uint32), want)
    b.set_layout(gr.LAYOUT_BVH8_Q8)
    b.trace_device(d_rays, m, d_hits)
    torch.cuda.synchronize()
    np.testing.assert_array_equal(d_hits.cpu().numpy().view(np.uint32), want)
    b.close()
    ctx.close()


def test_nodes_grow_where_two_arrays_do_not_fit(oracle):
    """A rebuild with more triangles on a GPU with room for the larger node array in the smaller one's place, not beside it
    (everything else that the rebuild needs has grown before, but for the triangle array)."""
    import torch
    ctx = gr.Context(0)
    n, m = 2000000, 1400000
    v = sc.triangle_soup(n, seed_salt=886)
    verts = torch.from_numpy(v).cuda()
    rays = sc.incoherent_rays(1000, seed_salt=887)
    d_rays, d_hits = torch.from_numpy(rays).cuda(), torch.zeros(1000, 4, dtype=torch.float32, device="cuda")
    tree = oracle.lbvh(v)
    nodes, tris = oracle.bvh8(tree)
    other = gr.BVH(ctx)
    other.set_layout(gr.LAYOUT_BVH8_Q8)
    other.build_device(verts, n)  # the context's memory for 8-wide builds
    other.close()
    b = gr.BVH(ctx)
    b.build_device(verts, n)
    b.build_device(verts, m)
    b.set_layout(gr.LAYOUT_BVH8_Q8)
    small, small_tris = b.layout_size(gr.LAYOUT_BVH8_Q8)
    grow_tris = tris.nbytes - small_tris
    assert nodes.nbytes > small > (16 << 20)
    held = fill_gpu(grow_tris + nodes.nbytes - small // 2)
    try:
        b.build_device(verts, n)
        b.trace_device(d_rays, 1000, d_hits)
        torch.cuda.synchronize()
    finally:
        del held
        torch.cuda.empty_cache()
    np.testing.assert_array_equal(b.export_layout(gr.LAYOUT_BVH8_Q8), nodes)
    np.testing.assert_array_equal(d_hits.cpu().numpy().view(np.uint32), oracle.trace(tree, rays).view(np.uint32))
    b.close()
    ctx.close()
