"""Single terms of the judge's exact repulsion (gvizCudaForceExactRepulsion),
held to the exact value of the reference's expression over the whole range of
distances that doubles hold.

A straight-line term is r = reciprocal(fl(dx^2)) to 2^-52, then fl(r dx). With
one coordinate equal the relative error is at most 2^-53 for the square, 2^-52
for the reciprocal and 2^-53 for the product: 2^-51. Every other source is so
far that its term is less than half an ulp of the sum, so adding it changes
nothing. Outside the straight-line range (squares below 2^-900 or from 2^1022)
the term is the reference's own expression, a square, a root and two
divisions, each to half an ulp, and two products: 2^-50 where the square is a
normal number."""
from fractions import Fraction

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

N = 96  # sources 32..63 and 64..95 are whole chunks that do not hold the target


def _term(dx, far, model=1, edge=10.0):
    """force on vertex 0 of a source at distance dx, everyone else at ~far"""
    from grapher_b200 import ForceLayout
    lay = ForceLayout(np.zeros(N + 1, np.uint64), np.zeros(0, np.uint32), model=model)
    lay.set_params(edgeLength=edge)
    p = np.zeros((N, 2))
    p[1:, 0] = far * (1.0 + np.arange(1, N) / 1024.0)
    p[40] = [dx, 0.0]
    lay.set_positions(p.reshape(-1))
    got = lay.exact_repulsion(np.zeros(1, np.uint32))[0]
    lay.close()
    return got


def _relative(got, want):
    return abs(Fraction(got) / want - 1)


@pytest.mark.parametrize("model", [0, 1])
def test_reciprocal_over_its_range(model):
    """Random mantissas at distances from 2^-449 to 2^440 (squares 2^-898 to
    2^880), the others at 2^60 times the distance."""
    rng = np.random.default_rng(4 + model)
    worst = Fraction(0)
    for e in list(range(-449, 440, 13)) + [-449, -2, -1, 0, 1, 2, 440]:
        for m in rng.uniform(1.0, 2.0, 2):
            dx = float(np.ldexp(m, e))
            got = _term(dx, float(np.ldexp(1.0, e + 66)), model)
            want = Fraction(-100 if model == 0 else -1) / Fraction(dx)
            worst = max(worst, _relative(got[0], want))
            assert got[1] == 0.0
    assert worst <= Fraction(1, 2 ** 51) * (2 if model == 0 else 1)  # FR: the product with k^2


def test_largest_distances():
    """Every source near the upper end: 95 comparable terms. 2^-51 of each, and
    at most 96 additions of half an ulp of the sum: 2^-51 + 96 * 2^-53."""
    for e in (500, 509, 510):
        far = float(np.ldexp(1.0, e))
        got = _term(far * 0.75, far)
        dist = [far * (1.0 + j / 1024.0) for j in range(1, N)]
        dist[39] = far * 0.75
        want = -sum(Fraction(1) / Fraction(d) for d in dist)
        assert _relative(got[0], want) <= Fraction(1, 2 ** 51) + Fraction(96, 2 ** 53)


@pytest.mark.parametrize("scale", [1.0, 2.0 ** -448, 2.0 ** -452, 2.0 ** -505, 2.0 ** -511])
def test_terms_below_the_range(scale):
    """distances whose squares are normal numbers, on both sides of 2^-900"""
    dx = 1.375 * scale
    got = _term(dx, 1.0 if scale < 1.0 else 2.0 ** 80)
    assert _relative(got[0], Fraction(-1) / Fraction(dx)) <= Fraction(1, 2 ** 50)


@pytest.mark.parametrize("model", [0, 1])
@pytest.mark.parametrize("dx", [2.0 ** -512, 1e-155, 1e-160, 3e-162])
def test_squares_below_the_normal_range(dx, model):
    """the reference's distance is the root of a subnormal square: finite, of
    the size of 1 / distance, never infinite"""
    want = (100.0 if model == 0 else 1.0) / np.sqrt(dx * dx)
    got = _term(dx, 1.0, model)
    # dirx = dx / dist, mag = num / dist
    assert abs(got[0] + want * (dx / np.sqrt(dx * dx))) <= 4 * np.spacing(want)
    assert got[1] == 0.0


def test_squares_above_the_range():
    """a squared distance that overflows gives no force; one just below does"""
    big = 2.0 ** 511.5
    got = _term(big, 1.5 * big)
    dist = [1.5 * big * (1.0 + j / 1024.0) for j in range(1, N)]
    dist[39] = big
    want = -sum(Fraction(1) / Fraction(d) for d in dist if d * d != np.inf)
    assert any(d * d == np.inf for d in dist)
    assert _relative(got[0], want) <= Fraction(1, 2 ** 50) + Fraction(96, 2 ** 53)
