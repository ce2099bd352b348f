"""The plain FP32 walk's rounds against exact FP64 repulsion: with a tiny
opening threshold every term is a pair term (even the smallest cells, of half
size 1e-9 around coincident points, stay open), so the walk must give the
all-pairs sum, at task edges (32 targets), with exactly coincident points (a
round's guarded path) and with and without radii.

Tolerance: a term carries a few FP32 roundings and one approximate reciprocal
or reciprocal square root (about 5e-7 of it), a round's plain partial at most
32 roundings (2e-6 of its terms); the compensated sum adds none. The positions
are multiples of 1/64, exact in the walk's split coordinates, and apart by at
least that much or not at all. Over the vertices the errors act at random, so
1e-5 of the RMS force bounds the RMS error."""
import numpy as np
import pytest

from helpers import cfg, make_layout

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [2, 31, 32, 33, 64, 65, 257, 1500])
@pytest.mark.parametrize("model", [0, 1])
@pytest.mark.parametrize("overlap", [False, True])
def test_all_pairs_when_nothing_is_accepted(n, model, overlap):
    from grapher_b200 import graphs
    a, b = graphs.random_connected(n, 0.0, 3)
    row, col = graphs.to_csr(n, a, b)
    # pairs 1/64 apart at the closest stay clear of the radii's contact
    lay = make_layout(row, col, cfg(model=model, theta=1e-12, prevent_overlap=overlap,
                                    radius_base=2.0 ** -9 if overlap else 0.0))
    cells = np.random.default_rng(n).choice(1 << 24, n, replace=False)
    x0 = np.stack([cells >> 12, cells & 4095], 1).astype(np.float64).reshape(-1) / 64.0
    if n > 60:
        x0[2 * 40:2 * 50] = x0[:20]  # coincident points
    lay.begin(0, positions=x0)
    lay.step()
    lay.set_positions(x0)
    got, want = lay.repulsion(), lay.exact_repulsion(np.arange(n))
    lay.close()
    assert np.sqrt(np.mean((got - want) ** 2)) <= 1e-5 * np.sqrt(np.mean(want ** 2))
