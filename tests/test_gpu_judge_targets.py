"""gvizCudaForceExactRepulsion keeps its workspace from call to call: lists of
other targets and other lengths in turn, on one handle, must give what a fresh
handle gives, bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _layout(n):
    from grapher_b200 import ForceLayout, graphs
    a, b = graphs.random_connected(n, 0.0, 5)
    lay = ForceLayout(*graphs.to_csr(n, a, b), model=1)
    lay.set_positions(graphs.randomize_positions(n, 100.0, 9))
    return lay


@pytest.mark.parametrize("n", [300, 20000])
def test_lists_of_changing_length(n):
    rng = np.random.default_rng(n)
    lists = [rng.permutation(n)[:m].astype(np.uint32)
             for m in (1, n, 7, 129, n // 2, 3, 128, n, 1)]
    kept = _layout(n)
    for t in lists:
        got = kept.exact_repulsion(t)
        fresh = _layout(n)
        want = fresh.exact_repulsion(t)
        fresh.close()
        assert np.array_equal(got, want)
    kept.close()
