"""GRIP rounds against a plain restatement in Python floats (IEEE doubles, the
reference's operation order, src/embedders/gvizGRIPEmbedder.c:870-1334): with
strict reductions bit for bit over several rounds, at list lengths around the
force kernel's lanes and batches, layers of a few vertices and of more than a
block; with the default sums within 1e-12 of the extent (sums of at most a few
thousand doubles in another order)."""
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

EDGE = 10.0


def _round(state, layer, active, off, kv, kd, row, col):
    pos, disp, heat, cos, calc = state
    force = {}
    for i, v in enumerate(active):
        px, py = pos[v]
        fx = fy = 0.0
        if layer == 0:
            for u in col[row[v]:row[v + 1]]:
                dx, dy = pos[u][0] - px, pos[u][1] - py
                d2 = dx * dx + dy * dy
                if d2 < 1e-18:
                    continue
                s = d2 / (EDGE * EDGE)
                fx += s * dx
                fy += s * dy
        for e in range(off[i], off[i + 1]):
            u = kv[e]
            if layer > 0:
                L = float(kd[e]) * EDGE
                if L < 1e-9:
                    continue
                dx, dy = pos[u][0] - px, pos[u][1] - py
                s = math.sqrt(dx * dx + dy * dy) / L - 1.0
            else:
                dx, dy = px - pos[u][0], py - pos[u][1]
                d2 = dx * dx + dy * dy
                if d2 < 1e-18:
                    continue
                s = 0.05 * (EDGE * EDGE) / d2
            fx += s * dx
            fy += s * dy
        ox, oy = disp[v]
        h = heat[v]
        n = math.sqrt(fx * fx + fy * fy)
        if not calc[v]:
            calc[v] = True
            h = EDGE / 6.0
        else:
            on = math.sqrt(ox * ox + oy * oy)
            if not (abs(n) < 1e-7 or abs(on) < 1e-7):
                c = (fx * ox + fy * oy) / (n * on)
                h *= (1 + c * 0.15 * 3) if c > 0 and cos[v] > 0 else (1 + c * 0.15)
                cos[v] = c
        h = max(min(h, EDGE * 10), EDGE * 1e-4)
        if n > 1e-7:
            s = h / n
            fx *= s
            fy *= s
        force[v] = n
        heat[v] = h
        disp[v] = (fx, fy)
    sx = sy = cx = cy = 0.0
    for v in active:
        sx += disp[v][0]
        sy += disp[v][1]
        cx += pos[v][0]
        cy += pos[v][1]
    count = float(len(active))
    mx, my = sx * (1.0 / count), sy * (1.0 / count)
    cx, cy = cx / count, cy / count
    L = I = 0.0
    for v in active:
        dx, dy = disp[v][0] + -1.0 * mx, disp[v][1] + -1.0 * my
        rx, ry = pos[v][0] - cx, pos[v][1] - cy
        L += rx * dy - ry * dx
        I += rx * rx + ry * ry
    rotate = len(active) >= 3 and not abs(I) < 1e-7
    w = L / I if rotate else 0.0
    top = total = 0.0
    for v in active:
        dx, dy = disp[v][0] + -1.0 * mx, disp[v][1] + -1.0 * my
        if rotate:
            rx, ry = pos[v][0] - cx, pos[v][1] - cy
            dx -= 0.0 * 0.0 - w * ry
            dy -= w * rx - 0.0 * 0.0
        disp[v] = (dx, dy)
        pos[v] = (pos[v][0] + 1.0 * dx, pos[v][1] + 1.0 * dy)
        n = math.sqrt(dx * dx + dy * dy)
        top = max(top, n)
        total += n
    force_sum = heat_sum = 0.0  # (Python's sum() compensates its rounding)
    for v in active:
        heat_sum += heat[v]
        force_sum += force[v]
    return [top, total / len(active), force_sum / len(active), heat_sum / len(active)]


@pytest.mark.parametrize("V,active,k,layer", [
    (2, 2, 1, 0), (40, 3, 2, 1), (60, 60, 5, 0), (200, 33, 4, 2), (200, 200, 17, 0),
    (400, 129, 31, 3), (400, 400, 16, 1), (700, 700, 40, 0)])
@pytest.mark.parametrize("strict", [True, False])
def test_rounds_match_a_plain_restatement(V, active, k, layer, strict):
    from grapher_b200 import graphs
    from grapher_b200.grip import GripRefiner, k_nearest
    a, b = graphs.random_connected(V, 0.02, 3)
    row, col = graphs.to_csr(V, a, b)
    rng = np.random.default_rng(V + k)
    act = rng.permutation(V)[:active].astype(np.uint32)
    seen = np.zeros(V, np.uint8)
    seen[act] = 1
    off, kv, kd = k_nearest(row, col, act, k, visible=seen)
    x0 = rng.uniform(-50.0, 50.0, (V, 2))
    if V > 100:
        x0[act[1]] = x0[act[0]]  # two active vertices at one place
    g = GripRefiner(row, col)
    g.set_strict_reductions(strict)
    g.set_positions(x0.reshape(-1))
    assert np.array_equal(g.positions(), x0.reshape(-1))
    g.set_layer(layer, act, off, kv, kd)
    state = ([tuple(map(float, p)) for p in x0], [(0.0, 0.0)] * V, [0.0] * V, [0.0] * V,
             [False] * V)
    lists = [x.astype(np.int64).tolist() for x in (act, off, kv, kd, row, col)]
    for _ in range(3):
        want = _round(state, layer, *lists)
        got = g.refine_round()
        pos = g.positions()
        heat, disp, cos = g.decorators()
        ref = np.array(state[0]).reshape(-1)
        if strict:
            assert np.array_equal(pos, ref)
            assert np.array_equal(got, np.array(want))
            assert np.array_equal(heat, np.array(state[2]))
            assert np.array_equal(disp, np.array(state[1]).reshape(-1))
            assert np.array_equal(cos, np.array(state[3]))
        else:
            assert np.abs(pos - ref).max() <= 1e-12 * 100.0
            assert np.allclose(got, want, rtol=1e-11, atol=0)
    g.close()
