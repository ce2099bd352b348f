"""Quadtree membership (bit-exact against the oracle) at the sizes where the
build's kernels change shape: the edges of a sort tile, of the rule that
picks the tile, and of a block."""
import numpy as np
import pytest

from test_gpu_tree import point_layout

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 2, 31, 33, 255, 256, 257, 1023, 1024, 1025, 2047, 2048, 2049, 4096, 4097, 131072, 131073])
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


def _nested_chains(structures, cluster, seed):
    """`structures` chains of 40 nested cells, three single points beside each,
    ending in a dense cluster: every chain node spans the whole cluster."""
    rng = np.random.default_rng(seed)
    j = 2.0 ** np.arange(19, -21, -1)
    ring = np.concatenate([j[:, None] * np.array(c) for c in
                           [(0.75, 0.25), (0.25, 0.75), (0.75, 0.75)]])
    out = []
    for k in range(structures):
        o = 2.0 ** 20 * np.array([k % 8, k // 8])
        core = rng.integers(0, 2 ** 8, (cluster, 2)) * 2.0 ** -28
        out.append(o + np.concatenate([ring, core]))
    return np.concatenate(out)


@pytest.mark.parametrize("structures,cluster", [(80, 400), (32, 3900)])
@pytest.mark.parametrize("k", [1, 3])
def test_many_nodes_above_blocks(oracle, structures, cluster, k):
    """Many nodes spanning blocks of 256 buckets, and spanning the wider ranges
    above those: with 32 chains more than the kernels that sum them hold in
    shared memory, so that they are worked off in global memory."""
    from test_gpu_tree import check_cells
    pts = _nested_chains(structures, cluster, 5)
    mass = 1.0 + (np.arange(len(pts)) % 5).astype(np.float64)
    od, ohi, olo, _ = oracle.quadtree_leaves(pts, mass, k)
    lay = point_layout(pts, mass, k)
    d, hi, lo, _ = lay.tree_leaves()
    nodes = lay.tree_nodes()
    lay.close()
    assert np.array_equal(d, od)
    assert np.array_equal(hi, ohi) and np.array_equal(lo, olo)
    check_cells(nodes, oracle.quadtree_nodes(pts, mass, k), float(np.abs(pts).max()))


def test_forest_above_blocks(oracle):
    """Graphs from one point to several super-ranges side by side."""
    rng = np.random.default_rng(8)
    sizes = [3, 300, 1, 5000, 4096, 12000, 255, 257, 1]
    pts = [rng.normal(0, 10.0, (n, 2)) for n in sizes]
    offs = np.concatenate([[0], np.cumsum(sizes)]).astype(np.uint64)
    allp = np.concatenate(pts)
    lay = point_layout(allp, np.ones(len(allp)), 2, graph_offsets=offs)
    d, hi, lo, _ = lay.tree_leaves()
    lay.close()
    for g, p in enumerate(pts):
        od, ohi, olo, _ = oracle.quadtree_leaves(p, np.ones(len(p)), 2)
        s = slice(int(offs[g]), int(offs[g + 1]))
        assert np.array_equal(d[s], od) and np.array_equal(hi[s], ohi) and np.array_equal(lo[s], olo)


@pytest.mark.parametrize("n", [(1 << 20) + 1, (1 << 22) + 1])
def test_membership_of_large_layouts(oracle, n):
    """Just above the sizes at which the ranges above blocks grow."""
    rng = np.random.default_rng(n)
    pts = rng.normal(0, 100.0, (n, 2))
    pts[: n // 3] *= 1e-3
    mass = np.ones(n)
    od, ohi, olo, _ = oracle.quadtree_leaves(pts, mass, 1)
    lay = point_layout(pts, mass, 1)
    d, hi, lo, _ = lay.tree_leaves()
    lay.close()
    assert np.array_equal(d, od)
    assert np.array_equal(hi, ohi) and np.array_equal(lo, olo)
