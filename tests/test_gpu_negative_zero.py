"""A coordinate of -0.0 is on the same side of a cell's centre as +0.0 (the
reference compares p >= c): a layout centred on the origin whose zeros are
negated, as a flipped axis makes them, has the same tree and the same step."""
import numpy as np
import pytest

from helpers import cfg, csr_of, make_layout
from test_gpu_tree import check_cells, point_layout

pytestmark = pytest.mark.gpu


def _flipped_grid(side):
    """an odd grid centred on the origin, y flipped: its middle row is y = -0.0"""
    c = np.arange(side) - side // 2
    x, y = np.meshgrid(c.astype(np.float64), -(c.astype(np.float64)))
    return np.stack([x.reshape(-1), y.reshape(-1)], 1)


def _cases():
    yield "grid3", _flipped_grid(3)
    yield "grid33", _flipped_grid(33)
    yield "grid129", _flipped_grid(129)  # more points than one sort block takes
    g = _flipped_grid(33)
    yield "turned", -g  # both axes: the centre is (-0.0, 0.0)
    zeros = np.array([[0.0, 0.0], [-0.0, 0.0], [0.0, -0.0], [-0.0, -0.0]])
    yield "coincident", np.concatenate([g, np.tile(zeros, (20, 1))])
    # points beside the origin that share the sorted bits of their paths, so
    # that the whole path is taken
    near = np.array([[s * 1e-8, z] for s in (1, -1, 2, -2) for z in (0.0, -0.0)])
    yield "near", np.concatenate([g, zeros, near, near[:, ::-1]])


@pytest.mark.parametrize("k", [1, 3])
@pytest.mark.parametrize("case", [c[0] for c in _cases()])
def test_membership_matches_oracle(oracle, case, k):
    pts = dict(_cases())[case]
    assert np.any((pts == 0) & np.signbit(pts))
    mass = 1.0 + (np.arange(len(pts)) % 5).astype(np.float64)
    od, ohi, olo, _ = oracle.quadtree_leaves(pts, mass, k)
    for forest in (False, True):
        if forest:  # the same points as the second of two graphs
            lay = point_layout(np.concatenate([pts[:2] + 5.0, pts]),
                               np.concatenate([[1.0, 1.0], mass]), k,
                               graph_offsets=np.array([0, 2, 2 + len(pts)], np.uint64))
        else:
            lay = point_layout(pts, mass, k)
        d, hi, lo, _ = lay.tree_leaves()
        nodes = lay.tree_nodes()
        lay.close()
        s = 2 if forest else 0
        assert np.array_equal(d[s:], od)
        assert np.array_equal(hi[s:], ohi) and np.array_equal(lo[s:], olo)
        if not forest:
            check_cells(nodes, oracle.quadtree_nodes(pts, mass, k), float(np.abs(pts).max()))


@pytest.mark.parametrize("precision", ["fp32", "fp64"])
@pytest.mark.parametrize("model", [0, 1])
def test_step_is_that_of_positive_zeros(precision, model):
    from grapher_b200 import graphs
    a, b = graphs.grid(33, 33)
    row, col = csr_of(33 * 33, a, b)
    out = []
    for pts in (_flipped_grid(33), _flipped_grid(33) + 0.0):
        lay = make_layout(row, col, cfg(model=model, theta=0.7, precision=precision, gravity=1.0))
        lay.begin(0, positions=pts.reshape(-1))
        lay.step()
        out.append((lay.positions(), lay.forces()["structForce"]))
        lay.close()
    assert np.array_equal(out[0][0], out[1][0])
    assert np.array_equal(out[0][1], out[1][1])
