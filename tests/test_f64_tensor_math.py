"""The accuracy check of the FP64 contraction on the tensor cores, restated in Python integers:
wherever sum_k p_a p_b >= 20 N holds, the truncated product of eight balanced base-256 digits is
within 4 2^-53 sum_k |a_k| |b_k| of the exact one (csrc/split.cu, launch_f64_tensor)."""
from fractions import Fraction

import numpy as np
import pytest

S = 8


def digits(row):
    """(exponent, digits of every element) with |x| < 2^e, most significant first."""
    mx = max((abs(x) for x in row), default=0.0)
    e = int(np.frexp(mx)[1]) if mx > 0 else 0
    out = []
    for x in row:
        num = Fraction(x) * Fraction(2) ** (7 + 8 * (S - 1) - e)
        F = round(num)  # ties to even
        assert abs(F) < 2 ** 63 or mx == 0
        d = []
        for _ in range(S - 1):
            low = ((F + 127) % 256) - 127
            d.append(low)
            F = (F - low) >> 8
        assert -128 <= F <= 128
        out.append([F] + d[::-1])
    return e, out


def check_and_error(a, b):
    eA, A = digits(a)
    eB, B = digits(b)
    R = sum(x[s] * y[t] * 2 ** (8 * (S - 1 - s - t)) for x, y in zip(A, B) for s in range(S) for t in range(S - s))
    got = Fraction(R) * Fraction(2) ** (eA + eB - 14 - 8 * (S - 1))
    exact = sum(Fraction(x) * Fraction(y) for x, y in zip(a, b))
    mag = sum(abs(Fraction(x)) * abs(Fraction(y)) for x, y in zip(a, b))
    n = sum(1 for x, y in zip(a, b) if x != 0 and y != 0)
    margin = sum(max(abs(x[0]) - 1, 0) * max(abs(y[0]) - 1, 0) for x, y in zip(A, B)) - 20 * n
    bound = Fraction(9.04) * Fraction(2) ** (eA + eB - 64) * n
    assert abs(got - exact) <= bound
    # the magnitudes the check sums are lower bounds
    for v, e, dg in ((a, eA, A), (b, eB, B)):
        for x, d in zip(v, dg):
            assert max(abs(d[0]) - 1, 0) <= 128 * abs(Fraction(x)) / Fraction(2) ** e
    return margin >= 0, abs(got - exact), Fraction(4) * Fraction(2) ** -53 * mag


ROWS = {
    "normal": lambda r, k: r.standard_normal(k),
    "uniform": lambda r, k: r.uniform(-1, 1, k),
    "decaying": lambda r, k: r.standard_normal(k) * np.exp(-0.1 * np.arange(k)),
    "graded up": lambda r, k: r.standard_normal(k) * 10.0 ** np.linspace(-8, 8, k),
    "graded down": lambda r, k: r.standard_normal(k) * 10.0 ** np.linspace(8, -8, k),
    "sparse": lambda r, k: r.standard_normal(k) * (r.random(k) < 0.1),
    "one large": lambda r, k: np.concatenate([[1e12], r.standard_normal(k - 1)]),
    "zero": lambda r, k: np.zeros(k),
    "subnormal": lambda r, k: r.standard_normal(k) * 5e-320,
    "integers": lambda r, k: r.integers(-128, 129, k).astype(float),
}


@pytest.mark.parametrize("left", sorted(ROWS))
@pytest.mark.parametrize("right", sorted(ROWS))
def test_check_implies_bound(left, right):
    rng = np.random.default_rng(len(left) * 100 + len(right))
    for k in (32, 75):
        for _ in range(3):
            ok, err, limit = check_and_error([float(x) for x in ROWS[left](rng, k)], [float(x) for x in ROWS[right](rng, k)])
            assert not ok or err <= limit


def test_ordinary_rows_pass_the_check():
    rng = np.random.default_rng(0)
    for kind in ("normal", "uniform", "decaying", "integers"):
        for k in (75, 300):
            assert check_and_error([float(x) for x in ROWS[kind](rng, k)], [float(x) for x in ROWS[kind](rng, k)])[0]


def test_opposed_grading_fails_the_check():
    rng = np.random.default_rng(1)
    a, b = ([float(x) for x in ROWS[n](rng, 60)] for n in ("graded up", "graded down"))
    ok, err, limit = check_and_error(a, b)
    assert not ok and err > limit
