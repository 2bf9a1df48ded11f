"""Registers whose coefficients use the whole 96-bit normal form, which
ab_write_register takes: their forward transforms, and products whose result is
in range, against Python integers, in the passes (a thread per word and a thread
per group) and in the resident runs."""
import random

import numpy as np
import pytest

import annie_b200 as A
import ntt_model
from helpers import PRIMES
from test_gpu_resident import PCK, _number

pytestmark = pytest.mark.gpu


def _words(K, exact):
    """The reference's register words of exact coefficient values."""
    return np.array([v % PRIMES[k] for k in range(K) for v in exact], dtype=np.uint32)


def _edges(K):
    """Values at the ends of the normal form (of 3 primes: those of their product)."""
    if K == 3:
        top = (PRIMES[0] * PRIMES[1] * PRIMES[2] - 1) // 2
        return [top, -top, 1 << 91, -(1 << 91) - 1, (1 << 94) - 1]
    return [(1 << 95) - 1, -(1 << 95), 1 << 91, -(1 << 91) - 1, (1 << 95) - (1 << 63), (1 << 92) + 12345, -(1 << 94)]


def _value(K, v):
    """The value that the words of v have in the reference's normal form: its
    leading mixed-radix digit is balanced (ocl/kernel.cl:1231-1470), so just above
    -P/2 the range of 3 primes ends a little earlier than at the other side."""
    p, q = PRIMES[0], PRIMES[1] * PRIMES[2]
    return v + p * q if K == 3 and v < -(p // 2) * q else v


@pytest.mark.parametrize("K,lbase,ln,row_levels", [(3, 20, 8, 0), (4, 27, 7, 0), (5, 17, 6, 0), (5, 17, 10, 4), (4, 27, 13, 11)])
def test_forward_of_the_whole_range(K, lbase, ln, row_levels):
    params = (K, PCK[K], ln, lbase)
    t = A.Transform(_number(params, ln), 3, params=params)
    if row_levels:
        t.set_geometry(row_levels)
    n, rng = 1 << ln, random.Random(K)
    lim = _edges(K)[0]
    x = [rng.randrange(-lim, lim) for _ in range(n)]
    for i, v in enumerate(_edges(K)):
        x[i] = x[n - 1 - i] = v
    for dom in (0, 1):
        got = t.diag_forward(_words(K, x), dom).astype(np.uint64)
        for k in range(K + 1):
            p = ntt_model.TPRIMES[k]
            res = np.array([_value(K, v) % p for v in x], dtype=np.uint64)
            exp = ntt_model.forward(res, ln, k, dom == 1, reduce_out=True) % p
            assert np.array_equal(got[k * n:(k + 1) * n] % p, exp), "domain %d, prime %d" % (dom, k)


@pytest.mark.parametrize("K,lbase,ln,row_levels", [(3, 20, 6, 0), (4, 27, 9, 0), (5, 17, 6, 0), (5, 17, 12, 0),
                                                   (5, 17, 8, 5), (5, 17, 10, 4), (4, 27, 13, 11), (4, 27, 13, 6)])
def test_product_by_a_register_of_the_whole_range(K, lbase, ln, row_levels):
    # get = value / (R/2) mod N and mul = x y / (R/2) mod N; row_levels: the
    # passes with that split, 0 the default path (resident)
    params = (K, PCK[K], ln, lbase)
    N, W, n = _number(params, ln + 1), PCK[K] * lbase, 1 << ln
    t = A.Transform(N, 3, params=params)
    if row_levels:
        t.set_geometry(row_levels)
    scale = pow((pow(2, W * n, N) - 1) * pow(2, -1, N), -2, N)
    for shift in (0, 1, n // 2 + 3):
        for v in _edges(K):
            x = [0] * n
            x[n - 5], x[3] = v, 7
            y = [0] * n
            y[shift] = 1
            t.write_register(0, _words(K, x))
            t.write_register(1, _words(K, y))
            t.mul(0, 1)
            X, Y = (_value(K, v) << W * (n - 5)) + (7 << 3 * W), 1 << shift * W
            assert t.get(0) == X * Y * scale % N, "value %x, shift %d" % (v, shift)
