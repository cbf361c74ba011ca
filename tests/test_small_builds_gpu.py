"""LBVH builds around the sizes where the bottom-up pass changes hands: one chunk of
256 positions, one sort tile, the one-block climb's spread and its largest size,
with runs of equal codes across chunk borders.
Trees against the oracle, word for word."""
import numpy as np
import pytest

import gr
from gr import scenes as sc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [255, 256, 257, 512, 513, 4096, 4097, 16384, 16385, 131071, 131072, 131073])
@pytest.mark.parametrize("runs", [False, True])
def test_trees_match_oracle(ctx, oracle, n, runs):
    v = sc.triangle_soup(n, seed_salt=n)
    if runs:  # equal codes: a run over a third of the positions, and one of two in every hundred
        v[n // 3:2 * n // 3] = v[n // 3]
        v[::100] = v[min(1, n - 1)]
    b = gr.BVH(ctx)
    b.build_host(v)
    got, want = b.export(), oracle.lbvh(v)
    assert got["root"] == want["root"]
    for k in ("sorted_prim", "sorted_code", "nodes", "ref_nodes"):
        np.testing.assert_array_equal(got[k], want[k], err_msg=k)
    np.testing.assert_array_equal(got["tris"].view(np.uint32), want["tris"].view(np.uint32))
    b.close()


@pytest.mark.parametrize("n", [1, 511, 512, 513, 1024, 1025, 1537, 2049, 2561, 3072, 3073, 5121, 65536, 65537, 98304, 98305,
                               131073, 155648, 155649, 233472, 233473, 389121, 466945, 544769, 622592, 622593, 933889,
                               1089537, 1245184, 1245185])
def test_sort_tiles_match_oracle(ctx, oracle, n):
    """At the sizes where the sort's tiles grow from 512 to 4,096 keys (one tile, up to 64, one an SM, all resident) and
    where it leaves the cooperative launch: order and codes against the oracle, with runs of equal codes."""
    v = sc.triangle_soup(n, seed_salt=n)
    v[::7] = v[n // 2]
    b = gr.BVH(ctx)
    b.build_host(v)
    got, want = b.export(), oracle.lbvh(v)
    for k in ("sorted_prim", "sorted_code", "nodes"):
        np.testing.assert_array_equal(got[k], want[k], err_msg=k)
    b.close()
