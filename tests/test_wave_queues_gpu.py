"""The wave's queues at their edges: depths of one and no bounce, single pixels,
queues shorter than a warp and just past a block, alone and packed with scenes
of other depths. Each image against the oracle's (the bound of the other image
tests), and the packed render bit for bit against the same scenes alone."""
import numpy as np
import pytest

import gr
from gr import scenes as sc

pytestmark = pytest.mark.gpu


def _mre(img, ref):
    floor = 0.01 * max(float(np.mean(ref)), 1e-6)
    return float(np.mean(np.abs(img - ref) / np.maximum(np.abs(ref), floor)))


@pytest.mark.parametrize("layout", [gr.LAYOUT_BVH2, gr.LAYOUT_BVH8_Q8])
@pytest.mark.parametrize("w,h,spp,depth", [(1, 1, 1, 1), (31, 1, 1, 2), (33, 9, 1, 0), (43, 6, 3, 17), (257, 5, 2, 5)])
def test_short_queues_match_oracle_alone_and_packed(ctx, oracle, layout, w, h, spp, depth):
    descs = [sc.glossy_scene(w, h, level=2, glass_level=1), sc.cornell_box(w + 2, h), sc.textured_scene(w, h + 1)]
    depths = [depth, depth + 2, max(depth - 1, 0)]
    alone = []
    for d, dep in zip(descs, depths):
        s = gr.Scene(ctx, d)
        s.set_tuning(layout, 64, 12)
        img, st = s.render(spp, max_depth=dep, seed=11)
        assert st.device_errors == 0
        ref = oracle.render(d, spp, max_depth=dep, seed=11) / float(spp)
        assert _mre(img, ref) < 1e-3
        alone.append((s.accumulation()[0], st.closest_rays, st.shadow_rays))
        s.close()
    packed = [gr.Scene(ctx, d) for d in descs]
    for s in packed:
        s.set_tuning(layout, 64, 12)
    st = gr.render_batch(ctx, packed, [dict(spp=spp, max_depth=dep, seed=11) for dep in depths])
    for s, (want, _, _) in zip(packed, alone):
        np.testing.assert_array_equal(s.accumulation()[0], want)
        s.close()
    assert st.closest_rays == sum(a[1] for a in alone) and st.shadow_rays == sum(a[2] for a in alone)


@pytest.mark.parametrize("layout", [gr.LAYOUT_BVH2, gr.LAYOUT_BVH8_Q8])
@pytest.mark.parametrize("w,h,spp", [(512, 256, 2), (511, 257, 2), (512, 257, 2)])
def test_material_groups_and_queue_order_render_the_same(ctx, layout, w, h, spp):
    """Waves of 2^18 paths and a few more (shaded in queue order up to there, in material groups above), against the same render cut into small waves, and with a scene of other materials in the wave: bit for bit."""
    desc, other = sc.glossy_scene(w, h, level=3, glass_level=2), sc.textured_scene(64, 48)
    got = []
    for wave_paths in (0, w * h):
        s = gr.Scene(ctx, desc)
        s.set_tuning(layout, 64, 12)
        _, st = s.render(spp, max_depth=9, seed=5, wave_paths=wave_paths)
        assert st.device_errors == 0
        got.append((s.accumulation()[0], st.closest_rays, st.shadow_rays))
        s.close()
    assert got[0][1:] == got[1][1:]
    np.testing.assert_array_equal(got[0][0], got[1][0])
    packed = [gr.Scene(ctx, d) for d in (desc, other)]
    for s in packed:
        s.set_tuning(layout, 64, 12)
    gr.render_batch(ctx, packed, [dict(spp=spp, max_depth=9, seed=5)] * 2)
    np.testing.assert_array_equal(packed[0].accumulation()[0], got[0][0])
    for s in packed:
        s.close()
