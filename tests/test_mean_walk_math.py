"""The walk of the impulse-accumulation means (CPU, exact integers): the sum of
many splines over a span is carried from its Taylor coefficients at an anchor
sample to the samples on either side, its third-order coefficient changed at
every knot's row, as the kernels do it (forwards: the step, then the jump at the
row reached; backwards: the jump at the row left taken back, then the step)."""
from fractions import Fraction

import numpy as np
import pytest


def spline(rng, lo, hi):
    """A piecewise cubic with integer coefficients about its first knot, continuous to the second order: knots x and the
    pieces' third-order coefficients, and its value at any sample."""
    x = np.unique(rng.integers(lo, hi, rng.integers(2, 14)))
    d = [int(v) for v in rng.integers(-2 ** 40, 2 ** 40, len(x))]
    a, b, c = (int(v) for v in rng.integers(-2 ** 50, 2 ** 50, 3))

    def taylor(n):  # value, slope, half the second derivative and third-order coefficient at n (the piece holding n)
        t = n - int(x[0])
        out = [a + b * t + c * t * t + d[0] * t ** 3, b + 2 * c * t + 3 * d[0] * t * t, c + 3 * d[0] * t, d[0]]
        for j in range(1, len(x)):
            u = n - int(x[j])
            if u >= 0:  # the piece from x_j on
                jump = d[j] - d[j - 1]
                out = [out[0] + jump * u ** 3, out[1] + 3 * jump * u * u, out[2] + 3 * jump * u, out[3] + jump]
        return out

    return x, d, taylor


@pytest.mark.parametrize("rows,anchor,seed", [(8, 4, 0), (32, 16, 1), (64, 32, 2), (31, 16, 3), (5, 4, 4), (1, 0, 5)])
def test_walk_from_the_anchor_is_the_sum_of_the_splines(rows, anchor, seed):
    rng = np.random.default_rng(seed)
    p0 = 100
    envs = [spline(rng, p0 - 40, p0 + rows + 40) for _ in range(37)]
    jumps = [0] * rows
    for x, d, _ in envs:
        for j in range(1, len(x)):
            if p0 < x[j] < p0 + rows:
                jumps[x[j] - p0] += d[j] - d[j - 1]
    A, B, C, D = (sum(t(p0 + anchor)[i] for _, _, t in envs) for i in range(4))
    got = {anchor: A}
    a, b, c, d = A, B, C, D
    for r in range(anchor + 1, rows):
        a, b, c = a + b + c + d, b + 2 * c + 3 * d, c + 3 * d
        d += jumps[r]
        got[r] = a
    a, b, c, d = A, B, C, D
    for r in range(anchor, 0, -1):
        d -= jumps[r]
        a, b, c = a + c - b - d, b + 3 * d - 2 * c, c - 3 * d
        got[r - 1] = a
    assert [got[r] for r in range(rows)] == [sum(t(p0 + r)[0] for _, _, t in envs) for r in range(rows)]


def nearest(v):
    return v.numerator / v.denominator if v else 0.0  # correctly rounded


@pytest.mark.parametrize("seed", range(4))
def test_quotient_by_a_rounded_reciprocal_is_the_division(seed):
    """(sum / 2) / Q of the FP64 mean: the product with the correctly rounded
    reciprocal and one correction by the exact remainder (Markstein 1990)."""
    rng = np.random.default_rng(seed)
    for q in [1, 2, 3, 7, 1023, 1024] + [int(v) for v in rng.integers(1, 65537, 60)]:
        rq = Fraction(nearest(Fraction(1, q)))
        near = [nearest(Fraction(k, 1) * q + s * Fraction(1, 2)) for k in (2 ** 52 + 1, 2 ** 53 - 1) for s in (-1, 0, 1)]
        for v in [float(x) for x in rng.standard_normal(40) * 2.0 ** rng.integers(-300, 300, 40)] + near:
            v = Fraction(v)
            q0 = Fraction(nearest(v * rq))
            rem = Fraction(nearest(v - q0 * q))
            assert nearest(q0 + rem * rq) == nearest(v / q)


@pytest.mark.parametrize("seed", range(3))
def test_last_place_of_a_reciprocal_from_the_low_product_word(seed):
    """FP64 pivots: of the three doubles about 1 / a, the one whose mantissa Y
    leaves 2 |2^105 - A Y| <= A, had from the low 64 bits of A Y, is 1 / a
    rounded to nearest; each of its neighbours is moved onto it."""
    rng = np.random.default_rng(seed)
    values = [3.0, 4.0, 5.0, 1024.0, 2.0 ** 20 - 1, float(np.nextafter(4.0, 5.0)), float(np.nextafter(8.0, 7.0))]
    for a in values + [float(v) for v in 3.0 + rng.random(2000) * 2.0 ** rng.integers(0, 24, 2000)]:
        right = nearest(1 / Fraction(a))
        A = (int(np.float64(a).view(np.int64)) & (2 ** 52 - 1)) | 2 ** 52
        for y in (np.nextafter(right, 0.0), right, np.nextafter(right, 1.0)):
            Y = int(np.float64(y).view(np.int64))
            r2 = ((-A * ((Y & (2 ** 52 - 1)) | 2 ** 52)) * 2) & (2 ** 64 - 1)
            r2 -= 2 ** 64 if r2 >= 2 ** 63 else 0
            Y += (r2 > A) - (r2 < -A)
            if A == 2 ** 52 and y < right:
                continue  # (a power of two: the step itself is exact, and a binade's lower neighbour half as far)
            assert float(np.int64(Y).view(np.float64)) == right, a
