"""The FP64 path's sums do not depend on how its kernels share the work: rows
of any length add their attraction terms in row order, bit for bit, and a
graph's walk gives the same bits alone (few targets per warp) and in a forest
large enough for full warps."""
import numpy as np
import pytest

from helpers import cfg, make_layout

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("degree", [1, 15, 16, 17, 31, 32, 33, 64, 100, 4096, 4097])
def test_attraction_adds_in_row_order(degree):
    from grapher_b200 import ForceLayout
    # vertex 0's row, in a scrambled order; everyone else has no row
    rng = np.random.default_rng(degree)
    n = degree + 1
    row = np.full(n + 1, degree, np.uint64)
    row[0] = 0
    col = (1 + rng.permutation(degree)).astype(np.uint32)
    x = rng.normal(0.0, 100.0, (n, 2))
    if degree > 20:
        x[col[7]] = x[0]  # a neighbour at no distance: no term
    lay = ForceLayout(row, col, model=0)
    lay.set_params(precision=1, barnesHutEnabled=0)
    lay.begin(0, positions=x.reshape(-1))
    lay.step()
    got = lay.forces()["attMag"][0]
    lay.close()
    ax = ay = np.float64(0.0)
    for u in col:
        dx, dy = x[u] - x[0]
        dist = np.sqrt(dx * dx + dy * dy)
        if dist < 1e-9:
            continue
        s = dist / 10.0
        ax += s * dx
        ay += s * dy
    assert got == np.sqrt(ax * ax + ay * ay)


@pytest.mark.parametrize("model", [0, 1])
def test_walk_is_the_same_alone_and_in_a_forest(model):
    from grapher_b200 import graphs
    sizes = [700, 13000, 1, 30000, 9001]
    parts = [(n,) + graphs.random_connected(n, 0.0, 3 + n) for n in sizes]
    row, col, offs = graphs.batch(parts)
    x0 = [graphs.randomize_positions(n, 80.0, n) for n in sizes]
    c = cfg(model=model, theta=0.7, precision="fp64", gravity=1.0)
    forest = make_layout(row, col, c, graph_offsets=offs)
    forest.begin(0, positions=np.concatenate(x0))
    forest.step()
    got = forest.forces()["structForce"]
    forest.close()
    for g, (n, a, b) in enumerate(parts):
        r, k = graphs.to_csr(n, a, b)
        lay = make_layout(r, k, c)
        lay.begin(0, positions=x0[g])
        lay.step()
        want = lay.forces()["structForce"]
        lay.close()
        assert np.array_equal(got[2 * int(offs[g]):2 * int(offs[g + 1])], want), n


@pytest.mark.parametrize("model", [0, 1])
@pytest.mark.parametrize("n", [700, 5921, 11841, 23681])
def test_listed_terms_add_in_walk_order(n, model):
    """At every number of targets per warp below 32 the walk lists its terms and
    helper lanes compute them; with 32 each lane adds its own as it goes. The
    same bits, with a dense core whose lists fill several times, coincident
    points and radii."""
    from grapher_b200 import graphs
    x = graphs.randomize_positions(n, 80.0, n).reshape(-1, 2)
    x[: n // 4] *= 1e-3
    x[n // 2: n // 2 + 5] = x[n // 2]
    big = 48000  # with this graph beside it every warp holds 32 targets
    parts = [(n,) + graphs.random_connected(n, 0.0, 3 + n),
             (big,) + graphs.random_connected(big, 0.0, 4)]
    row, col, offs = graphs.batch(parts)
    c = cfg(model=model, theta=0.3, precision="fp64", gravity=1.0, prevent_overlap=True,
            radius_base=0.01)
    forest = make_layout(row, col, c, graph_offsets=offs)
    forest.begin(0, positions=np.concatenate([x.reshape(-1),
                                              graphs.randomize_positions(big, 80.0, 1)]))
    forest.step()
    want = forest.forces()["structForce"][:2 * n]
    forest.close()
    r, k = graphs.to_csr(*parts[0])
    lay = make_layout(r, k, c)
    lay.begin(0, positions=x.reshape(-1))
    lay.step()
    got = lay.forces()["structForce"]
    lay.close()
    assert np.all(np.isfinite(want))
    assert np.array_equal(got, want)
