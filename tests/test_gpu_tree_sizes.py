"""Quadtree membership (bit-exact against the oracle) at the sizes where the
build's kernels change shape: the edges of a sort tile, of the rule that
picks the tile, and of a block."""
import numpy as np
import pytest

from test_gpu_tree import point_layout

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 2, 31, 33, 255, 256, 257, 1023, 1024, 1025, 2047, 2048, 2049, 4097, 131072, 131073])
@pytest.mark.parametrize("k", [1, 3])
def test_membership_at_tile_edges(oracle, n, k):
    rng = np.random.default_rng(n)
    pts = rng.normal(0, 100.0, (n, 2))
    pts[: n // 3] *= 1e-3  # a dense core
    pts[n // 2: n // 2 + n // 8] = pts[: n // 8]  # duplicates
    mass = 1.0 + (np.arange(n) % 3).astype(np.float64)
    od, ohi, olo, _ = oracle.quadtree_leaves(pts, mass, k)
    lay = point_layout(pts, mass, k)
    d, hi, lo, _ = lay.tree_leaves()
    lay.close()
    assert np.array_equal(d, od)
    assert np.array_equal(hi, ohi) and np.array_equal(lo, olo)
