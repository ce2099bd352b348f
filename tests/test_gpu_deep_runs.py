"""More than 4,096 distinct points in one of the smallest sorted cells are an
error (GVIZ_CUDA_ERR_DEEP_RUN) of every call that builds the tree; no kernel
walks keys that are not sorted, and the handle then works as a fresh one."""
import numpy as np
import pytest

from grapher_b200._native import GvizCudaError
from helpers import cfg, make_layout

pytestmark = pytest.mark.gpu

CORNERS = [(-1.0, 1.0), (0.31, -0.27), (1.0, -1.0)]  # first, inside and last in tree order


def _points(n, dense, corner, seed=3):
    rng = np.random.default_rng(seed)
    pts = rng.uniform(-1.0, 1.0, (n, 2)) * 1e6
    at = rng.permutation(n - 2)[:dense] + 2
    pts[0], pts[1] = (-1e6, -1e6), (1e6, 1e6)
    pts[at] = np.array(corner) * 0.999e6 + rng.uniform(-1e-4, 1e-4, (dense, 2))
    return pts


def _fails(call):
    with pytest.raises(GvizCudaError) as e:
        call()
    assert e.value.code == -7


@pytest.mark.parametrize("corner", CORNERS)
@pytest.mark.parametrize("precision", ["fp32", "fp64"])
@pytest.mark.parametrize("n,dense,before", [(4100, 4097, 0), (9000, 4097, 0), (9000, 4097, 300),
                                            (20000, 15000, 0), (150000, 120000, 5000)])
def test_error_and_recovery(n, dense, before, corner, precision):
    """before: vertices of two other graphs ahead of the dense one"""
    offs = np.array([0, 2, before, n], np.uint64) if before else None
    pts = np.concatenate([np.random.default_rng(1).normal(0, 1, (before, 2)),
                          _points(n - before, dense, corner)])
    row, col = np.zeros(n + 1, np.uint64), np.zeros(0, np.uint32)
    c = cfg(model=1, theta=0.8, precision=precision)
    lay = make_layout(row, col, c, graph_offsets=offs)
    lay.begin(0, positions=pts.reshape(-1))
    xy = pts.reshape(-1).copy()
    _fails(lay.step)
    _fails(lambda: lay.step_host(xy))
    _fails(lambda: lay.run(3, 0.0))
    _fails(lay.tree_leaves)
    _fails(lay.tree_nodes)
    _fails(lay.repulsion)
    good = np.random.default_rng(5).normal(0.0, 10.0, 2 * n)
    fresh = make_layout(row, col, c, graph_offsets=offs)
    out = []
    for h in (lay, fresh):
        h.begin(0, positions=good)
        h.step()
        h.step()
        out.append((h.positions(), h.forces()["structForce"], h.tree_leaves()[1]))
        h.close()
    for a, b in zip(*out):
        assert np.array_equal(a, b)


def test_learned_walk_reports_the_error():
    from grapher_b200.farfield import FarFieldModel
    pts = _points(20000, 15000, CORNERS[1])
    lay = make_layout(np.zeros(20001, np.uint64), np.zeros(0, np.uint32), cfg(model=1))
    m = FarFieldModel()
    m.attach(lay)
    lay.begin(0, positions=pts.reshape(-1))
    for groups in (0, 1):
        lay.set_params(farField=1, farCellGroups=groups, farHubTargets=64, farHubTheta=0.5)
        _fails(lay.step)
        _fails(lay.judge_far_field)
    good = np.random.default_rng(5).normal(0.0, 10.0, 40000)
    lay.begin(0, positions=good)
    lay.step()
    assert np.all(np.isfinite(lay.positions()))
    lay.close()
    m.close()
