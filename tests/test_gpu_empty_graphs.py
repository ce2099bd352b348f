"""Batches that hold graphs without vertices, first, in the middle, side by side
and last: every graph's steps, statistics and stopping are those of the graph
alone, an empty one takes its steps as the reference's empty embedder does
(displacement 0, speed 1), and strict reductions agree."""
import numpy as np
import pytest

from helpers import cfg, make_layout

pytestmark = pytest.mark.gpu

SIZES = [0, 40, 0, 0, 2500, 1, 0]


def _batch(strict, precision="fp32", bh=True):
    from grapher_b200 import graphs
    parts = [(n,) + (graphs.random_connected(n, 0.0, 3 + n) if n > 1 else
                     (np.zeros(0, np.uint32), np.zeros(0, np.uint32))) for n in SIZES]
    row, col, offs = graphs.batch(parts)
    c = cfg(model=1, theta=0.8, gravity=1.0, strict=strict, precision=precision, bh=bh)
    lay = make_layout(row, col, c, graph_offsets=offs)
    x0 = [graphs.randomize_positions(n, 10.0, 5) for n in SIZES]
    lay.begin(0, positions=np.concatenate(x0))
    return lay, parts, x0, c, offs


@pytest.mark.parametrize("strict", [False, True])
@pytest.mark.parametrize("precision,bh", [("fp32", True), ("fp64", True), ("fp64", False)])
def test_steps_and_statistics(strict, precision, bh):
    from grapher_b200 import graphs
    lay, parts, x0, c, offs = _batch(strict, precision, bh)
    for _ in range(3):
        lay.step()
    rows = [(s.maxDisp, s.speed, s.meanAttractive, s.meanRepulsive) for s in lay.last_stats]
    pos = lay.positions()
    for g, (n, a, b) in enumerate(parts):
        hist = lay.stat_history(g)
        assert hist.shape[0] == 3, f"graph {g}"
        if n == 0:
            assert rows[g] == (0.0, 1.0, 0.0, 0.0)
            assert np.array_equal(hist[:, :4], np.tile([0.0, 1.0, 0.0, 0.0], (3, 1)))
            continue
        one = make_layout(*graphs.to_csr(n, a, b), c)
        one.begin(0, positions=x0[g])
        for _ in range(3):
            one.step()
        assert np.array_equal(hist, one.stat_history(0)), f"graph {g}"
        assert np.array_equal(pos[2 * int(offs[g]):2 * int(offs[g + 1])], one.positions())
        one.close()
    lay.close()


@pytest.mark.parametrize("strict", [False, True])
def test_run_stops_and_counts_every_graph(strict):
    from grapher_b200 import graphs
    lay, parts, x0, c, _ = _batch(strict)
    # a displacement this large ends every graph after its first round ...
    assert lay.run(400, 1e9) == 1
    assert np.array_equal(lay.rounds, np.ones(len(SIZES), np.uint64))
    # ... and without a threshold an empty graph, which never moves more than
    # that, still counts every round
    lay.run(5, 0.0)
    assert np.array_equal(lay.rounds, np.full(len(SIZES), 5, np.uint64))
    # a displacement of 0 is below any threshold: empty graphs stop at once
    lay.run(30, 1e-3)
    rounds = lay.rounds.copy()
    for g, n in enumerate(SIZES):
        if n == 0:
            assert rounds[g] == 1
    assert lay.stat_history(0).shape[0] == 7
    lay.close()


def test_all_graphs_empty():
    lay = make_layout(np.zeros(1, np.uint64), np.zeros(0, np.uint32), cfg(),
                      graph_offsets=np.zeros(4, np.uint64))
    lay.begin(0, positions=np.zeros(0))
    assert lay.step() == 0.0
    lay.close()
