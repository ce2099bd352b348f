"""The exact FP32 kernel against the FP64 exact repulsion at the edges of its
tiles, chunks, target groups and source ranges, for layouts and forests.

Tolerance: a term carries a few FP32 roundings and one approximate reciprocal
(about 4e-7 of it), a chunk's plain partial at most 64 roundings (4e-6 of its
terms); the compensated sum over chunks adds none. Over a layout's vertices
these act at random, so 1e-5 of the RMS force bounds the RMS error."""
import numpy as np
import pytest

from helpers import cfg, make_layout

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [2, 3, 63, 65, 127, 128, 129, 511, 512, 513, 2049, 5000])
@pytest.mark.parametrize("model", [0, 1])
def test_exact_f32_matches_f64(n, model):
    from grapher_b200 import graphs
    a, b = graphs.random_connected(n, 0.0, 3)
    row, col = graphs.to_csr(n, a, b)
    lay = make_layout(row, col, cfg(model=model, bh=False))
    x0 = graphs.randomize_positions(n, 50.0, n)
    if n > 60:
        x0[2 * 40:2 * 50] = x0[:20]  # coincident points: the guarded path
    lay.begin(0, positions=x0)
    lay.step()
    lay.set_positions(x0)
    got = lay.repulsion()
    want = lay.exact_repulsion(np.arange(n))
    lay.close()
    err = np.sqrt(np.mean((got - want) ** 2))
    assert err <= 1e-5 * np.sqrt(np.mean(want ** 2))


def test_exact_f32_forest_straddles_tiles():
    from grapher_b200 import graphs
    sizes = [1, 130, 513, 64, 700, 2]
    row, col, offs = graphs.batch([(n,) + graphs.random_connected(n, 0.0, 5 + n) for n in sizes])
    n = int(offs[-1])
    lay = make_layout(row, col, cfg(model=1, bh=False), graph_offsets=offs)
    x0 = graphs.randomize_positions(n, 50.0, 9)
    lay.begin(0, positions=x0)
    lay.step()
    lay.set_positions(x0)
    got, want = lay.repulsion(), lay.exact_repulsion(np.arange(n))
    lay.close()
    assert np.sqrt(np.mean((got - want) ** 2)) <= 1e-5 * np.sqrt(np.mean(want ** 2))
