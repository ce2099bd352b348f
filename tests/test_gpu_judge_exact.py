"""The judge's exact repulsion of listed targets against plain FP64 sums, at
the edges of its tiles, target blocks and source ranges, in forests, with
radii and with coincident points.

Tolerance: a term carries a handful of FP64 roundings (1e-15 of it) and the
sums of at most a few thousand terms a few hundred more at random: 1e-12 of
the sum of the terms' sizes bounds every target's error."""
import numpy as np
import pytest

from helpers import cfg, make_layout

pytestmark = pytest.mark.gpu


def _forces(p, t, lo, hi, mass, rad, model):
    d = p[lo:hi] - p[t]
    dist = np.linalg.norm(d, axis=1)
    use = (np.arange(lo, hi) != t) & (dist > 0)
    d, dist = d[use], dist[use]
    m, r = mass[lo:hi][use], rad[lo:hi][use]
    gap = dist - (rad[t] + r)
    num = 100.0 * np.floor(m) if model == 0 else mass[t] * m
    mag = np.where(gap > 0, num / np.where(gap > 0, gap, 1.0), num * 100.0)
    f = -(mag / dist)[:, None] * d
    return f.sum(0), np.abs(mag).sum()


@pytest.mark.parametrize("n,targets", [(1, 1), (2, 2), (127, 127), (129, 128), (1000, 129),
                                       (3000, 7), (5000, 1)])
@pytest.mark.parametrize("model", [0, 1])
@pytest.mark.parametrize("overlap", [False, True])
def test_judge_matches_plain_sums(n, targets, model, overlap):
    from grapher_b200 import graphs
    half = n // 3  # two graphs in one handle where there are enough vertices
    parts = [(half,) + graphs.random_connected(half, 0.0, 1),
             (n - half,) + graphs.random_connected(n - half, 0.0, 2)] if half > 1 else [
                 (n,) + graphs.random_connected(n, 0.0, 1)]
    row, col, offs = graphs.batch(parts)
    radius = 0.125 if overlap else 0.0
    lay = make_layout(row, col, cfg(model=model, prevent_overlap=overlap, radius_base=radius),
                      graph_offsets=offs if len(parts) > 1 else None)
    x = graphs.randomize_positions(n, 60.0, n)
    lay.set_positions(x)
    p = x.reshape(-1, 2)
    deg = np.diff(row).astype(np.float64)
    mass = np.ones(n) if model == 0 else 1.0 + deg
    t = np.random.default_rng(n).permutation(n)[:targets].astype(np.uint32)
    got = lay.exact_repulsion(t)  # before any step: the status starts clean
    lay.close()
    for k, v in enumerate(t):
        g = int(np.searchsorted(offs, v, side="right")) - 1
        want, size = _forces(p, int(v), int(offs[g]), int(offs[g + 1]), mass,
                             np.full(n, radius), model)
        assert np.abs(got[k] - want).max() <= 1e-12 * max(size, 1e-300)


def test_judge_coincident_points_repel():
    from grapher_b200 import ForceLayout
    lay = ForceLayout(np.zeros(4, np.uint64), np.zeros(0, np.uint32), model=1)
    lay.set_positions(np.array([1.0, 2.0, 1.0, 2.0, 5.0, 2.0]))
    f = lay.exact_repulsion(np.arange(3))
    lay.close()
    # the pair's terms are opposite, of size numer * C = 100; the third's is 1/4
    assert abs(np.linalg.norm(f[0] - [-0.25, 0.0]) - 100.0) <= 1e-10
    assert np.abs(f[0] + f[1] + [0.5, 0.0]).max() <= 1e-10


@pytest.mark.parametrize("scale", [1e-140, 1e-130, 1.0, 1e150, 9e153])
@pytest.mark.parametrize("model", [0, 1])
def test_judge_at_extreme_distances(scale, model):
    """Squared distances on both sides of the range whose reciprocals the
    straight-line terms take (2^-900 to 2^1022), in whole chunks and the rest."""
    from grapher_b200 import graphs
    n = 100
    row, col, _ = graphs.batch([(n,) + graphs.random_connected(n, 0.0, 1)])
    lay = make_layout(row, col, cfg(model=model))
    p = np.random.default_rng(3).uniform(0.0, 1.0, (n, 2)) * scale
    lay.set_positions(p.reshape(-1))
    mass = np.ones(n) if model == 0 else 1.0 + np.diff(row).astype(np.float64)
    got = lay.exact_repulsion(np.arange(n, dtype=np.uint32))
    lay.close()
    for v in range(n):
        want, size = _forces(p, v, 0, n, mass, np.zeros(n), model)
        assert np.abs(got[v] - want).max() <= 1e-12 * size
