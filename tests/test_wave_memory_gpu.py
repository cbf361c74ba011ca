"""What a wave's path state takes: 172 bytes a path, so that a wave size that the caller asks for and that fits at that
size is rendered, as one wave, to the same image as with room to spare (where the shading groups have their arrays)."""
import numpy as np
import pytest

import gr
from gr import scenes as sc
from test_failed_builds_gpu import fill_gpu

pytestmark = pytest.mark.gpu
W, H, SPP = 1024, 1024, 8
PATHS = W * H * SPP


@pytest.mark.parametrize("layout", [gr.LAYOUT_BVH2, gr.LAYOUT_BVH8_Q8])
def test_an_asked_wave_fits_in_172_bytes_a_path(layout):
    import torch
    ctx = gr.Context(0)  # its own: the pool starts empty
    s = gr.Scene(ctx, sc.glossy_scene(W, H, level=3, glass_level=2))  # several material types
    s.set_tuning(layout, 64, 12)
    s.render(1, max_depth=3, seed=4, want_image=False)  # kernels and graphs loaded, a small pool
    s.reset()
    held = fill_gpu(PATHS * 177)
    try:
        _, st = s.render(SPP, max_depth=3, seed=4, wave_paths=PATHS, want_image=False)
    finally:
        del held
        torch.cuda.empty_cache()
    assert st.waves == 1 and st.device_errors == 0
    tight, rays = s.accumulation()[0], (st.closest_rays, st.shadow_rays)
    s.close()
    ctx.close()
    ctx = gr.Context(0)
    s = gr.Scene(ctx, sc.glossy_scene(W, H, level=3, glass_level=2))
    s.set_tuning(layout, 64, 12)
    _, st = s.render(SPP, max_depth=3, seed=4, wave_paths=PATHS, want_image=False)
    assert st.waves == 1 and rays == (st.closest_rays, st.shadow_rays)
    np.testing.assert_array_equal(s.accumulation()[0], tight)
    s.close()
    ctx.close()
