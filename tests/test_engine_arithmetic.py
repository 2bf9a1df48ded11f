"""The engine's arithmetic at the ends of its ranges, in the numpy model
(tests/ntt_model.py) against Python integers: the encoder over the whole 96-bit
normal form, the pointwise product on every lazy representative, the CRT for the
largest values and representatives, and the digit sizes of the parameter rule."""
import itertools
import random

import numpy as np
import pytest

import annie_b200 as A
import ntt_model as M

LIMBS = [0, 1, 0x7fffffff, 0x80000000, 0xffffffff]
PCK = {2: 1, 3: 2, 4: 2, 5: 4}


@pytest.mark.parametrize("K", range(2, 6))
def test_encode_takes_every_exact_value(K):
    rng = random.Random(K)
    vals = [a | b << 32 | c << 64 for a, b, c in itertools.product(LIMBS, repeat=3)] + [rng.getrandbits(96) for _ in range(50)]
    vals = [v - (1 << 96) if v >> 95 else v for v in vals]
    factors = [[1] * (K + 1)] + [M.Consts(ln, K).s for ln in range(6, 23)]
    for s in factors:
        for k in range(K + 1):
            p = M.TPRIMES[k]
            w, ok = M.encode_weights(k, s[k])
            assert ok
            for v in vals:                                  # the sum as a signed number
                d = v & ((1 << 96) - 1)
                t = (d & M.M32) * w[0] + (d >> 32 & M.M32) * w[1] + ((d >> 64) - ((d >> 95) << 32)) * w[2]
                assert -(1 << 63) <= t < 1 << 63 and -p // 2 <= t >> 32 < 2 * p
            r = M.encode(vals, k, s=s[k])
            assert all(0 < int(x) < 4 * p and int(x) % p == s[k] * v % p for x, v in zip(r, vals))


@pytest.mark.parametrize("k", range(6))
def test_products_of_every_representative(k):
    p = M.TPRIMES[k]
    ends = [0, 1, p - 1, p, p + 1, 2 * p - 2, 2 * p - 1]
    x = np.array(list(itertools.product(ends, repeat=4)), dtype=np.uint64)
    x0, x1, y0, y1 = x.T
    for c in (1, 2, p // 2, p - 1):
        cm = np.uint64(c * (1 << 32) % p)
        for mul in (True, False):
            z0, z1 = (y0, y1) if mul else (x0, x1)
            r0, r1 = M.poly_product(x0, x1, z0, z1, mul, cm, p)
            i = pow(1 << 32, -1, p)
            for a0, a1, b0, b1, g0, g1 in zip(*([int(t) for t in v] for v in (x0, x1, z0, z1, r0, r1))):
                assert g0 < 2 * p and g1 < 2 * p
                assert g0 % p == (a0 * b0 + a1 * b1 * c) * i % p and g1 % p == (a0 * b1 + a1 * b0) * i % p


@pytest.mark.parametrize("K", range(2, 6))
def test_crt_of_the_largest_values(K):
    rng = random.Random(10 * K)
    top = 1 << (32 * K - 1)
    vals = [0, 1, -1, top - 1, -top, top - 12345, 1 - top] + [rng.randrange(-top, top) for _ in range(60)]
    for ln in range(6, 23):
        c = M.Consts(ln, K)
        base = [[v * pow(c.M // p * c.e[k] % p, -1, p) % p for v in vals] for k, p in enumerate(M.TPRIMES[:K + 1])]
        # the coordinates as they are, all in [p, 2p), the largest lazy words, mixed
        for pick in (lambda y, p: y, lambda y, p: y + p, lambda y, p: y + p * rng.getrandbits(1)):
            y = [np.array([pick(v, M.TPRIMES[k]) for v in base[k]], dtype=np.uint64) for k in range(K + 1)]
            cols = [sum(int(max(y[k])) * c.mk[k][j] for k in range(K + 1)) for j in range(K - 1)]
            assert max(cols, default=0) + (1 << 38) < 1 << 64
            got = M.crt(y, ln, K)
            assert got == vals, "ln %d" % ln
        # values from the largest words themselves
        y = [np.array([2 * M.TPRIMES[k] - 1], dtype=np.uint64) for k in range(K + 1)]
        v = sum(int(y[k][0]) * (c.M // M.TPRIMES[k]) * c.e[k] for k in range(K + 1)) % c.M
        v = v - c.M if 2 * v > c.M else v
        if abs(v) < c.M >> 18:
            assert M.crt(y, ln, K)[0] == (v + top) % (2 * top) - top


def test_rule_sizes_take_the_fixed_digit_form():
    # W = pck lbase reaches into the last of a digit's limbs for every size that
    # the parameter rule gives bases up to 100 (split_digit FULL), so that two
    # limbs pass the carry of the second phase on; larger bases also get smaller
    # digits (the general form)
    seen = set()
    bits = 2400.0
    while bits < 2.6e8:
        for a in (2, 3, 5, 7, 11, 13, 100, 1000, 2**31 - 1):
            (K, pck, ln, lbase), _ = A.probe((1 << int(bits)) | 1, a, gcd=False)
            W, nd = pck * lbase, {1: 1, 2: 2, 4: 3}[pck]
            assert W <= 32 * nd and (W // 32 == nd - 1 or a > 100)
            if W // 32 == nd - 1:
                assert 32 * K - 1 - 2 * W <= 63
            seen.add((a, K, lbase))
        bits *= 1.15
    assert len(seen) > 40
