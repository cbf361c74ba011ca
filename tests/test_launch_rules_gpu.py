"""Ray queries around the points where the number of rays a warp takes changes: 4-wide nodes at 8 lanes, and trees of one or
two levels, which always fill their warps. Hits against the oracle's of the same layout, bit for bit."""
import numpy as np
import pytest

import gr
from gr import scenes as sc

pytestmark = pytest.mark.gpu


def _oracle_hits(oracle, layout, tree, rays, any_hit):
    if layout == gr.LAYOUT_BVH2:
        return oracle.trace(tree, rays, any_hit=any_hit)
    if layout == gr.LAYOUT_BVH8_Q8:
        n8, t8 = oracle.bvh8(tree)
        return oracle.trace8(tree, n8, t8, rays, any_hit=any_hit)
    quant = layout == gr.LAYOUT_BVH4_Q8
    return oracle.trace4(tree, oracle.bvh4(tree, quant), quant, rays, any_hit=any_hit)


@pytest.mark.parametrize("layout,block", [(gr.LAYOUT_BVH4, 128), (gr.LAYOUT_BVH4_Q8, 64), (gr.LAYOUT_BVH4_Q8, 256)])
def test_4_wide_fills(ctx, oracle, layout, block):
    v = sc.triangle_soup(5000, seed_salt=101)
    b = gr.BVH(ctx)
    b.build_host(v)
    b.set_tuning(layout, block, 12)
    tree = oracle.lbvh(v)
    for any_hit, rays in ((False, sc.incoherent_rays(20000, seed_salt=102)), (True, sc.shadow_rays(20000, seed_salt=103))):
        want = _oracle_hits(oracle, layout, tree, rays, any_hit).view(np.uint32)
        for n in (1, 33, 2432, 2433, 4865, 19456, 19457, 20000):
            got = b.trace_host(rays[:n], any_hit=any_hit).view(np.uint32)
            np.testing.assert_array_equal(got, want[:n], err_msg=str(n))
    b.close()


@pytest.mark.parametrize("layout", [gr.LAYOUT_BVH2, gr.LAYOUT_BVH4, gr.LAYOUT_BVH4_Q8, gr.LAYOUT_BVH8_Q8])
@pytest.mark.parametrize("tris", [1, 2, 4, 5, 8, 9])
def test_flat_trees(ctx, oracle, layout, tris):
    r = np.random.default_rng(104 + tris)
    v = (0.7 * r.normal(size=(tris, 9))).astype(np.float32)
    b = gr.BVH(ctx)
    b.build_host(v)
    b.set_tuning(layout, 64, 12)
    tree = oracle.lbvh(v)
    rays = np.zeros((5000, 8), np.float32)
    rays[:, :3] = r.normal(size=(5000, 3)) * 2.0
    rays[:, 3:6] = r.normal(size=(5000, 3)) * 0.3 - rays[:, :3]
    rays[:, 7] = 1e30
    for any_hit in (False, True):
        want = _oracle_hits(oracle, layout, tree, rays, any_hit).view(np.uint32)
        for n in (1, 33, 5000):
            np.testing.assert_array_equal(b.trace_host(rays[:n], any_hit=any_hit).view(np.uint32), want[:n])
    b.close()
