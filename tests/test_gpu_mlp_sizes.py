"""Mini-batches at the edges of the training kernels' 128-sample tiles, and the
fused gradient sum + Adam update, against the update formula over the gradients
that the library itself returns."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

MASK = (1 << 64) - 1
B1, B2, EPS, LR = np.float32(0.9), np.float32(0.999), 1e-8, 2e-3


def _order(n, seed):
    """The training call's seeded permutation (Fisher-Yates over splitmix64)."""
    s = (seed ^ 0xD1B54A32D192ED03) & MASK
    order = list(range(n))
    for i in range(n - 1, 0, -1):
        s = (s + 0x9E3779B97F4A7C15) & MASK
        z = s
        z = ((z ^ (z >> 30)) * 0xBF58476D1CE4E5B9) & MASK
        z = ((z ^ (z >> 27)) * 0x94D049BB133111EB) & MASK
        j = (z ^ (z >> 31)) % (i + 1)
        order[i], order[j] = order[j], order[i]
    return np.array(order)


@pytest.mark.parametrize("tc", [True, False], ids=["tcgen05", "mma_sync"])
@pytest.mark.parametrize("weighted", [True, False], ids=["weights", "unit"])
@pytest.mark.parametrize("n", [1, 127, 128, 129, 4097])
def test_two_steps_follow_the_update_formula(n, weighted, tc):
    """A rounding of powf(0.999, 2) is 3e-5 of the second moment's correction,
    1.5e-5 of the update, whose size is below 2 lr: 5e-5 lr in all, and one
    rounding of the weight."""
    from grapher_b200.farfield import FarFieldModel
    rng = np.random.default_rng(n)
    net, ref = FarFieldModel(seed=3), FarFieldModel(seed=3)
    for k in (net, ref):
        k.set_training_kernels(tc)
    w = ref.weights().astype(np.float64)
    m = v = 0.0
    for step in (1, 2):
        X = rng.uniform(-0.5, 0.5, (n, 10)).astype(np.float32)
        T = rng.uniform(-0.2, 0.2, (n, 2)).astype(np.float32)
        W = rng.uniform(0.1, 2.0, n).astype(np.float32) if weighted else None
        o = _order(n, 11 + step)
        ref.set_weights(net.weights())
        loss, g = ref.gradient(X[o], T[o], None if W is None else W[o])
        got = net.train(X, T, W, epochs=1, batch=n, lr=LR, seed=11 + step)
        assert abs(got[0] - loss) <= 1e-6 * loss
        g = g.astype(np.float64)
        m = float(B1) * m + float(np.float32(1) - B1) * g
        v = float(B2) * v + float(np.float32(1) - B2) * g * g
        c1, c2 = (float(np.float32(1) - b ** np.float32(step)) for b in (B1, B2))
        want = w - LR * (m / c1) / (np.sqrt(v / c2) + EPS)
        now = net.weights().astype(np.float64)
        real = now != 0.0
        assert np.count_nonzero(real) > 4000
        assert np.all(np.abs(now - want)[real] <= 5e-5 * LR + 1.2e-7 * np.abs(want[real]))
        w = now


@pytest.mark.parametrize("batch", [100, 128, 256, 1000])
def test_short_last_batch_is_deterministic(batch):
    from grapher_b200.farfield import FarFieldModel
    rng = np.random.default_rng(5)
    X = rng.uniform(-0.5, 0.5, (1000 + batch // 2, 10)).astype(np.float32)
    T = rng.uniform(-0.2, 0.2, (len(X), 2)).astype(np.float32)
    out = []
    for _ in range(2):
        net = FarFieldModel(seed=3)
        losses = net.train(X, T, None, epochs=3, batch=batch, lr=LR, seed=1)
        out.append((losses, net.weights()))
    assert np.all(np.isfinite(out[0][0]))
    assert np.array_equal(out[0][0], out[1][0]) and np.array_equal(out[0][1], out[1][1])
