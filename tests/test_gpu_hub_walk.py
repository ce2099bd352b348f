"""The hub targets' walk beside the learned walk (few hubs, small layouts) or
after it, on the two sides of the rule that picks: the same positions, to the
bit, as with every kernel in order."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# hubs times vertices: far below 2^28, just below, just above
@pytest.mark.parametrize("V,hubs", [(3000, 1), (3000, 3000), (1 << 14, (1 << 14) - 1),
                                    (1 << 14, 1 << 14), ((1 << 14) + 1, 1 << 14)])
@pytest.mark.parametrize("groups", [0, 1])
def test_hub_walk_order_does_not_show(V, hubs, groups):
    from grapher_b200 import ForceLayout, graphs
    from grapher_b200.farfield import FarFieldModel
    a, b = graphs.barabasi_albert(V, 4, 7)
    row, col = graphs.to_csr(V, a, b)
    pos = graphs.randomize_positions(V, 1000.0, 7)
    out = []
    for in_order in (True, False):
        lay = ForceLayout(row, col, model=1)
        net = FarFieldModel(seed=3)
        net.attach(lay)
        lay.set_params(theta=1.1, gravityK=1.0, preventOverlap=0, farField=1,
                       farCellGroups=groups, farHubTargets=hubs)
        lay.begin(0, positions=pos)
        for _ in range(4):
            if in_order:
                lay.profile_step()
            else:
                lay.step()
        out.append(lay.positions())
        lay.close()
        net.close()
    assert np.all(np.isfinite(out[0]))
    assert np.array_equal(out[0], out[1])
