"""Images to host memory, which come in chunks of 2^18 pixels through two page-locked buffers: none, one, a chunk and a few
pixels, several and a remainder, larger and smaller in turn on one context; bit for bit against the sums over the counts."""
import numpy as np
import pytest

import gr
from gr import scenes as sc

pytestmark = pytest.mark.gpu


def test_chunks_and_remainders(ctx):
    import torch
    fresh = gr.Context(0)  # its buffers grow from nothing
    for w, h in ((7, 5), (513, 512), (64, 48), (1025, 769), (512, 512), (1024, 513)):
        s = gr.Scene(fresh, sc.cornell_box(w, h))
        host, _ = s.render(2, max_depth=3, seed=7)
        total, count = s.accumulation()
        want = (total * (1.0 / count[..., None].astype(np.float64))).astype(np.float32)
        np.testing.assert_array_equal(host, want.reshape(host.shape))
        s.reset()
        out = torch.zeros(h, w, 3, dtype=torch.float32, device="cuda")
        s.render(2, max_depth=3, seed=7, out=out)
        np.testing.assert_array_equal(host, out.cpu().numpy())
        s.close()
    fresh.close()
