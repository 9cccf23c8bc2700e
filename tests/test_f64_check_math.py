"""The accuracy check of the FP64 form for outputs of few products, restated: an output passes with
no product, with at least eight and M >= 20 N, or with two to seven and M >= 20 N + 256 (N products
that are not zero, M the sum of their leading magnitudes' products).  What the digits leave out is then below the roundings of a
chain of FMAs, and a check taken in K slices decides as the whole one does."""
from fractions import Fraction

import numpy as np
import pytest

from test_f64_tensor_math import S, digits

PER, FEW, MORE, CAP = 20, 8, 256, 1 << 22


def fails(n, excess):
    return n == 1 or (n > 1 and excess < (MORE if n < FEW else 0))


def product(a, b):
    """(truncated product, exact product, magnitudes, N, M) of two rows."""
    (eA, A), (eB, B) = digits(a), digits(b)
    R = sum(x[s] * y[t] * 2 ** (8 * (S - 1 - s - t)) for x, y in zip(A, B) for s in range(S) for t in range(S - s))
    got = Fraction(R) * Fraction(2) ** (eA + eB - 14 - 8 * (S - 1))
    terms = [Fraction(x) * Fraction(y) for x, y in zip(a, b)]
    m = sum(max(abs(x[0]) - 1, 0) * max(abs(y[0]) - 1, 0) for x, y in zip(A, B))
    return got, sum(terms), sum(map(abs, terms)), sum(t != 0 for t in terms), m


def chain(a, b):
    s = Fraction(0)
    for x, y in zip(a, b):
        s = Fraction(float(Fraction(x) * Fraction(y) + s))
    return s


@pytest.mark.parametrize("n", [1, 2, 3, 4, 8, 32])
def test_few_products(n):
    rng = np.random.default_rng(n)
    ours, chains, passed = [], [], 0
    for q in range(400):
        more = MORE if n < FEW else 0
        size = 1.25 * np.sqrt(rng.uniform(20, 400) + more / n) / 128
        row = lambda: size * rng.uniform(0.4, 1.6, n) * rng.choice([-1, 1], n)
        a = np.concatenate([[0.99, 0.0], row()]).tolist()  # the largest elements meet zeros
        b = np.concatenate([[0.0, 0.99], row()]).tolist()
        got, exact, mag, N, M = product(a, b)
        assert N == n
        if fails(N, M - PER * N):
            continue
        passed += 1
        assert abs(got - exact) <= Fraction(9.04) * Fraction(2) ** -50 * N / (PER * N + more) * mag
        ours.append(float(abs(Fraction(float(got)) - exact) / mag))
        chains.append(float(abs(chain(a, b) - exact) / mag))
    if n == 1:
        assert passed == 0  # one product is rounded once by the FMA kernel
    else:
        assert passed > 50
        assert np.linalg.norm(ours) <= np.linalg.norm(chains)


def test_slices_decide_as_the_whole():
    pack = lambda n, excess: min(excess, CAP) * 16 + min(n, FEW)
    rng = np.random.default_rng(1)
    seen = set()
    for _ in range(20000):
        ks = int(rng.integers(1, 65))
        n = rng.integers(0, [2, 3, 6, 1025][rng.integers(0, 4)], ks) * (rng.random(ks) < rng.random())
        m = n * rng.integers(0, 128 * 128, ks) // [1, 8, 64, 512][rng.integers(0, 4)]
        if rng.random() < 0.3 and n.sum():  # near the line
            m = m * 0
            m[np.argmax(n)] = PER * n.sum() + (MORE if n.sum() < FEW else 0) + rng.integers(-2, 2)
        x = [pack(int(a), int(b - PER * a)) for a, b in zip(n, m)]
        whole = fails(int(n.sum()), int((m - PER * n).sum()))
        assert fails(sum(v & 15 for v in x), sum(v >> 4 for v in x)) == whole
        seen.add(whole)
    assert len(seen) == 2
