"""Ray queries whose rays do not fill the GPU's lanes: one ray, a warp's worth and
its neighbours, and counts around the points where the lanes a warp uses change.
Hits against the oracle's, bit for bit, closest and any hit, binary and 8-wide."""
import numpy as np
import pytest

import gr
from gr import scenes as sc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("layout,block", [(gr.LAYOUT_BVH2, 128), (gr.LAYOUT_BVH8_Q8, 64), (gr.LAYOUT_BVH8_Q8, 256)])
def test_hits_match_oracle_at_every_fill(ctx, oracle, layout, block):
    v = sc.triangle_soup(5000, seed_salt=71)
    b = gr.BVH(ctx)
    b.build_host(v)
    b.set_tuning(layout, block, 8)
    ob = oracle.lbvh(v)
    n8, t8 = oracle.bvh8(ob)
    inc, sh = sc.incoherent_rays(80000, seed_salt=72), sc.shadow_rays(80000, seed_salt=73)
    want = oracle.trace(ob, inc)
    want_any = oracle.trace(ob, sh, any_hit=True) if layout == gr.LAYOUT_BVH2 else oracle.trace8(ob, n8, t8, sh, any_hit=True)
    for n in (1, 2, 31, 32, 33, 1216, 2431, 2432, 2433, 4864, 4865, 40000, 75392, 77823, 77825, 80000):
        np.testing.assert_array_equal(b.trace_host(inc[:n]).view(np.uint32), want[:n].view(np.uint32), err_msg=str(n))
        np.testing.assert_array_equal(b.trace_host(sh[:n], any_hit=True).view(np.uint32), want_any[:n].view(np.uint32),
                                      err_msg=str(n))
    b.close()


@pytest.mark.parametrize("block", [64, 128, 256])
def test_hits_match_oracle_at_every_share_of_the_warps(ctx, oracle, block):
    """8-wide ray queries use between half and all of the resident warps: counts on
    both sides of each change (rays per resident lane 0.8, 1.3, 2.2, 3.2)."""
    v = sc.triangle_soup(3000, seed_salt=81)
    b = gr.BVH(ctx)
    b.build_host(v)
    b.set_tuning(gr.LAYOUT_BVH8_Q8, block, 12)
    ob = oracle.lbvh(v)
    inc = sc.incoherent_rays(520000, seed_salt=82)
    want = oracle.trace(ob, inc).view(np.uint32)
    for n in (77824, 110000, 124517, 124519, 202342, 202343, 342425, 342426, 498073, 498074, 520000):
        np.testing.assert_array_equal(b.trace_host(inc[:n]).view(np.uint32), want[:n], err_msg=str(n))
    b.close()
