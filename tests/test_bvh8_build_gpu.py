"""The 8-wide build where its launch and its arithmetic can go wrong: trees of one
to a few nodes, levels just around a warp's four nodes and a block's, rebuilds
that shrink and grow the kept node array, planes that fall exactly on a
quantisation step (lattices), and coordinates that are subnormal or huge. Nodes
and triangles against the oracle, word for word."""
import numpy as np
import pytest

import gr
from gr import scenes as sc

pytestmark = pytest.mark.gpu


def _check(b, oracle, v):
    b.build_host(v)
    want_nodes, want_tris = oracle.bvh8(oracle.lbvh(v))
    np.testing.assert_array_equal(b.export_layout(gr.LAYOUT_BVH8_Q8), want_nodes)
    np.testing.assert_array_equal(b.export_layout_tris(gr.LAYOUT_BVH8_Q8).view(np.uint32), want_tris.view(np.uint32))


@pytest.mark.parametrize("sizes", [(1, 2, 3, 8, 9, 10), (31, 33, 64, 65, 257), (20011, 700, 41000, 40999, 5)])
def test_sizes_and_rebuilds(ctx, oracle, sizes):
    b = gr.BVH(ctx)
    b.set_layout(gr.LAYOUT_BVH8_Q8)
    for n in sizes:
        _check(b, oracle, sc.triangle_soup(n, seed_salt=500 + n))
    b.close()


@pytest.mark.parametrize("name", ["lattice", "huge", "tiny", "subnormal"])
def test_planes_on_steps_and_extreme_coordinates(ctx, oracle, name):
    r = np.random.default_rng(77)
    v = sc.triangle_soup(3000, seed_salt=61).astype(np.float64)
    if name == "lattice":
        v = r.integers(0, 256, v.shape) / 16.0
    elif name == "huge":
        v = (v - 0.5) * 3.0e37
    elif name == "tiny":
        v = v * 1e-30
    elif name == "subnormal":
        v = v * 1e-40
    b = gr.BVH(ctx)
    b.set_layout(gr.LAYOUT_BVH8_Q8)
    f = np.ascontiguousarray(v, np.float32)
    _check(b, oracle, f)
    b.close()


@pytest.mark.parametrize("outer,inner", [(120, 3000), (200, 3000), (300, 9000)])
def test_levels_that_narrow_and_widen(ctx, oracle, outer, inner):
    """A loose soup, a chain towards a corner and a dense cluster in it: levels such as 1, 8, 56, 1, 8, 48, 316, 597, 6
    nodes, so the build passes from one block to all of them and back more than once."""
    chain = sc.triangle_soup(8, seed_salt=73).reshape(8, 9) * np.float32(2.0 ** -11)
    chain = chain + np.float32(2.0) ** -np.arange(1, 9, dtype=np.float32)[:, None]
    dense = sc.triangle_soup(inner, seed_salt=72) * np.float32(2.0 ** -9)
    v = np.concatenate([sc.triangle_soup(outer, seed_salt=71), chain, dense])
    b = gr.BVH(ctx)
    b.set_layout(gr.LAYOUT_BVH8_Q8)
    _check(b, oracle, np.ascontiguousarray(v, np.float32))
    _check(b, oracle, np.ascontiguousarray(v[::-1], np.float32))
    b.close()
