"""The carry of products whose digits are far smaller than their coefficients
(forced small digit sizes): carries beyond 64 and 96 bits between the
coefficients of a group, against the carry rule in Python integers, by a thread
per group, by four lanes per group, and in resident runs."""
import random

import numpy as np
import pytest

import annie_b200 as A
from helpers import PRIMES
from test_gpu_exact_range import _words
from test_gpu_resident import PCK, _number

pytestmark = pytest.mark.gpu


def _carry(V, W, nega):
    """The carry rule on groups of 4 coefficients: unsigned digits and the
    group's carry-out, then the carry-in with balanced digits, the last
    coefficient taking the rest."""
    n, half = len(V), 1 << (W - 1)
    d, out = [], []
    for i, v in enumerate(V):
        f = v + (f if i % 4 else 0)
        d.append(f % (1 << W))
        f >>= W
        if i % 4 == 3:
            out.append(f)
    x = []
    for i in range(n):
        if i % 4 == 0:
            c = out[i // 4 - 1] if i else (-out[-1] if nega else out[-1])
        s = d[i] + c
        c = 0 if i % 4 == 3 else (s + half) >> W
        x.append(s - (c << W))
    return x


# K, lbase, bits of the product's coefficients: carries into the second
# coefficient of a group of 2^(bits - 2 pck lbase), results of 96 bits at most
CASES = [(5, 10, 155), (5, 6, 144), (4, 8, 97), (4, 7, 92), (3, 7, 92)]


@pytest.mark.parametrize("row_levels", [4, 6, 7])
@pytest.mark.parametrize("K,lbase,bits", CASES)
def test_carry_of_large_coefficients(K, lbase, bits, row_levels):
    # 32 rows (a thread per group), 8 and 4 rows (four lanes per group)
    ln = 10
    params, W, n = (K, PCK[K], ln, lbase), PCK[K] * lbase, 1 << ln
    t = A.Transform(_number(params, bits), 3, params=params)
    t.set_geometry(row_levels)
    rng = random.Random(K * bits)
    xb = min(bits - 2, 93)
    y0 = rng.randrange(1 << (bits - xb - 1), 1 << (bits - xb)) if bits > xb + 1 else 1
    x = [rng.randrange(-(1 << xb), 1 << xb) if i % 4 == 3 else rng.randrange(-8, 8) for i in range(n)]
    y = [y0] + [0] * (n - 1)
    for dom in (0, 1):
        got = t.diag_product(_words(K, x), dom, 1, y=_words(K, y))
        exp = _words(K, _carry([v * y0 for v in x], W, dom == 1))
        assert np.array_equal(got, exp), "domain %d: %d words differ" % (dom, np.count_nonzero(got != exp))


@pytest.mark.parametrize("K,lbase,bits", CASES)
def test_product_with_large_coefficients_resident(K, lbase, bits):
    ln = 6
    params, W, n = (K, PCK[K], ln, lbase), PCK[K] * lbase, 1 << ln
    N = _number(params, bits + 1)
    t = A.Transform(N, 3, params=params)
    half = (pow(2, W * n, N) - 1) * pow(2, -1, N) % N
    xb = min(bits - 2, 93)
    for i, v in ((3, (1 << xb) + 99), (n - 1, -(1 << xb) + 5), (n // 2 + 3, 3 << (xb - 2))):
        y0 = 1 << max(0, bits - xb - 1)
        x, y = [0] * n, [0] * n
        x[i], y[0] = v, y0
        t.write_register(0, _words(K, x))
        t.write_register(1, _words(K, y))
        t.mul(0, 1)
        assert t.get(0) == (v * y0 << W * i) * pow(half, -2, N) % N, "coefficient %d" % i


def _square(x, B, nega):
    """Coefficients of x^2 mod x^n -+ 1, below 2^(B-1) in magnitude (by one product
    of integers with B bits per coefficient)."""
    n, half = len(x), 1 << (B - 1)
    X = sum(v << B * i for i, v in enumerate(x))
    p, c = X * X, []
    for _ in range(2 * n):
        d = ((p + half) & ((1 << B) - 1)) - half
        c.append(d)
        p = (p - d) >> B
    return [c[i] - c[i + n] if nega else c[i] + c[i + n] for i in range(n)]


# K, lbase, ln inside the parameter rule
EXTREME = [(2, 14, 10), (3, 21, 9), (3, 20, 12), (4, 28, 10), (4, 27, 11), (5, 18, 10), (5, 17, 11)]


def _extreme(K, lbase, ln):
    """Registers of extreme digits: all-maximal, the most negative balanced ones,
    both beside each other; and the largest multiplier that they leave room for."""
    W, n, P = PCK[K] * lbase, 1 << ln, 1
    for p in PRIMES[:K]:
        P *= p
    big, low = (1 << W) - 1, -(1 << (W - 1))
    a = min((1 << 31) - 1, P // 2 >> (ln + 2 * W))
    assert a >= 3
    return [[big] * n, [low] * n, [low, big] * (n // 2), [low] * (n - 1) + [big], [big] + [low] * (n - 1)], a


@pytest.mark.parametrize("rows", [5, 3, 1])
@pytest.mark.parametrize("K,lbase,ln", EXTREME)
def test_extreme_digits(K, lbase, ln, rows):
    # 32 rows (a thread per group), 8 and 2 rows (four lanes per group)
    params, W = (K, PCK[K], ln, lbase), PCK[K] * lbase
    t = A.Transform(_number(params, 3 * ln), 3, params=params)
    if ln - 1 - rows < 4:
        rows = ln - 5
    t.set_geometry(ln - 1 - rows)
    regs, amax = _extreme(K, lbase, ln)
    for x in regs:
        for dom in (0, 1):
            V = _square(x, 2 * W + ln + 3, dom == 1)
            for a in (1, amax):
                got = t.diag_product(_words(K, x), dom, a)
                assert np.array_equal(got, _words(K, _carry([a * v for v in V], W, dom == 1))), "domain %d, a = %d" % (dom, a)


@pytest.mark.parametrize("K,lbase,ln", EXTREME)
def test_extreme_digits_resident(K, lbase, ln):
    # up to about half of R, as a register of a number within the rule
    params, W, n = (K, PCK[K], ln, lbase), PCK[K] * lbase, 1 << ln
    N = _number(params, 3 * ln)
    t = A.Transform(N, 3, params=params)
    scale = pow((pow(2, W * n, N) - 1) * pow(2, -1, N), -2, N)
    regs, a = _extreme(K, lbase, ln)
    for x in regs:
        x = x[:n // 2] + [0] * (n - n // 2)
        X = sum(v << W * i for i, v in enumerate(x))
        t.write_register(0, _words(K, x))
        t.write_register(1, _words(K, x))
        t.square_mul(a)
        assert t.get(0) == a * X * X * scale % N
        t.mul(1, 1)
        assert t.get(1) == X * X * scale % N
