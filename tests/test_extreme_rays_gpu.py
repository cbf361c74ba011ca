"""Rays with NaN, infinite, zero and crossed fields, and vertices that are NaN or infinite: misses where no number can be
a hit, in no more time than ordinary rays take; hits, and the 8-wide nodes and triangles that the oracle collapses from
the same binary tree, bit for bit."""
import numpy as np
import pytest

import gr
from gr import scenes as sc

pytestmark = pytest.mark.gpu
NAN, INF = np.float32(np.nan), np.float32(np.inf)


def _misses(rays):
    """Miss records: t = the ray's tmax, triangle -1, no barycentrics."""
    want = np.zeros((len(rays), 4), np.float32)
    want[:, 0] = rays[:, 7]
    want.view(np.uint32)[:, 1] = 0xFFFFFFFF
    return want.view(np.uint32)


@pytest.mark.parametrize("any_hit", [False, True])
@pytest.mark.parametrize("layout", [gr.LAYOUT_BVH2, gr.LAYOUT_BVH4, gr.LAYOUT_BVH4_Q8, gr.LAYOUT_BVH8_Q8])
def test_intervals_without_a_number_miss(ctx, layout, any_hit):
    b = gr.BVH(ctx)
    b.build_host(sc.triangle_soup(4000, seed_salt=91))
    b.set_tuning(layout, 64, 12)
    rays = sc.incoherent_rays(7 * 64, seed_salt=92)
    rays[0:64, 6] = NAN
    rays[64:128, 7] = NAN
    rays[128:192, 6:8] = NAN
    rays[192:256] = NAN
    rays[256:320, 6], rays[256:320, 7] = 1.0, 0.5
    rays[320:384, 6] = INF
    rays[384:448, 3:6] = NAN  # an interval, but no direction
    np.testing.assert_array_equal(b.trace_host(rays, any_hit=any_hit).view(np.uint32), _misses(rays))
    b.close()


@pytest.mark.parametrize("any_hit", [False, True])
def test_nan_rays_do_not_walk_the_tree(ctx, any_hit):
    """4,096 rays of NaN take no longer than ten times as many ordinary ones (a walk over 300,007 triangles takes thousands
    of times as long)."""
    import torch
    n = 300007
    b = gr.BVH(ctx)
    b.build_host(sc.triangle_soup(n, seed_salt=93))
    b.set_tuning(gr.LAYOUT_BVH8_Q8, 64, 12)
    good = torch.from_numpy(sc.incoherent_rays(40960, seed_salt=94)).cuda()
    bad = torch.full((4096, 8), float("nan"), dtype=torch.float32, device="cuda")
    hits = torch.zeros(40960, 4, dtype=torch.float32, device="cuda")
    stream = torch.cuda.current_stream().cuda_stream

    def ms(rays):
        best = 1e30
        for _ in range(4):
            e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            e0.record()
            b.trace_device(rays, len(rays), hits, any_hit=any_hit, stream=stream)
            e1.record()
            e1.synchronize()
            best = min(best, e0.elapsed_time(e1))
        return best

    assert ms(bad) < ms(good)
    b.close()


def _extreme_rays(m, v):
    """Origins on vertices, triangles and around; directions with zero, huge and tiny components; tmax infinite; some NaN and
    infinite fields."""
    r = np.random.default_rng(95)
    tri = v.reshape(-1, 3, 3)[r.integers(0, len(v), m)]
    rays = np.zeros((m, 8), np.float32)
    w = np.where(r.random((m, 1)) < 0.5, r.dirichlet([1, 1, 1], m), np.eye(3)[r.integers(0, 3, m)])
    rays[:, :3] = np.einsum("mk,mkc->mc", w, tri)
    away = r.random(m) < 0.4
    rays[away, :3] = r.random((int(away.sum()), 3)) * 2.0 - 0.5
    d = r.normal(size=(m, 3))
    axis = r.integers(0, 3, m)
    one, two = r.random(m) < 0.4, r.random(m) < 0.2
    d[one, axis[one]] = 0.0
    d[two, (axis[two] + 1) % 3] = -0.0
    d /= np.maximum(np.linalg.norm(d, axis=1, keepdims=True), 1e-9)
    d *= r.choice([1.0, 1.0, 1.0, 1e-20, 1e20], m)[:, None]
    rays[:, 3:6] = d
    rays[:, 6] = r.choice(np.array([0, 0, -0.0, 1e-4, -1], np.float32), m)
    rays[:, 7] = r.choice(np.array([INF, INF, 1e34, 0.9999, -0.0], np.float32), m)
    k = m // 16
    rays[:k, 3] = NAN
    rays[k:2 * k, 0] = NAN
    rays[2 * k:3 * k, 4] = INF
    rays[3 * k:4 * k, 1] = -INF
    rays[4 * k:5 * k, 3:6] = 0.0
    return rays


@pytest.mark.parametrize("name", ["soup", "flat", "lattice"])
def test_extreme_rays_match_oracle(ctx, oracle, name):
    v = sc.triangle_soup(3000, seed_salt=96)
    if name == "flat":
        v = (v * np.array([1, 0, 1] * 3, np.float32)).astype(np.float32)
    elif name == "lattice":
        v = np.random.default_rng(97).integers(0, 8, (3000, 9)).astype(np.float32)
    rays = _extreme_rays(8192, v)
    tree = oracle.lbvh(v)
    n8, t8 = oracle.bvh8(tree)
    b = gr.BVH(ctx)
    b.build_host(v)
    for any_hit in (False, True):
        b.set_tuning(gr.LAYOUT_BVH2, 64, 12)
        want = oracle.trace(tree, rays, any_hit=any_hit)
        np.testing.assert_array_equal(b.trace_host(rays, any_hit=any_hit).view(np.uint32), want.view(np.uint32))
        b.set_tuning(gr.LAYOUT_BVH8_Q8, 64, 12)
        want = oracle.trace8(tree, n8, t8, rays, any_hit=any_hit)
        np.testing.assert_array_equal(b.trace_host(rays, any_hit=any_hit).view(np.uint32), want.view(np.uint32))
    b.close()


@pytest.mark.parametrize("name", ["nan", "nan_many", "inf", "inf_nan"])
def test_vertices_without_a_place_match_oracle(ctx, oracle, name):
    v = sc.triangle_soup(3000, seed_salt=98)
    if name == "nan":
        v[17, 3], v[400] = NAN, NAN
    elif name == "nan_many":
        v[::7] = NAN
    elif name == "inf":
        v[17, 3], v[911, 7] = INF, -INF
    else:
        v[::5, 1], v[::9, 2] = INF, NAN
    b = gr.BVH(ctx)
    b.build_host(v)
    tree = b.export()
    if "nan" not in name:  # where a NaN corner sorts is not the oracle's
        np.testing.assert_array_equal(tree["nodes"], oracle.lbvh(v)["nodes"])
    n8, t8 = oracle.bvh8(tree)
    b.set_layout(gr.LAYOUT_BVH8_Q8)
    np.testing.assert_array_equal(b.export_layout(gr.LAYOUT_BVH8_Q8), n8)
    np.testing.assert_array_equal(b.export_layout_tris(gr.LAYOUT_BVH8_Q8).view(np.uint32), t8.view(np.uint32))
    b.close()
