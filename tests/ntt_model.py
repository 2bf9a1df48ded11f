"""Bit-exact numpy model of the engine's own transform arithmetic (not the
reference's): the transform primes, the Shoup twiddle tables, the lazily
reduced butterflies, the summed Montgomery pointwise products, the image factors
and the radix-2^30 CRT with its 32-bit quotient estimate, level by level.  Every
element goes through the same operations in the same order as in the CUDA passes
(only the grouping of butterflies into passes differs), so the model reproduces
the device's lazy words; it is the reference for the forward-transform kernel test
and, on the CPU, checks the design against exact big-integer convolutions.
"""
import numpy as np

TPRIMES = [119 * (1 << 23) + 1, 107 * (1 << 23) + 1, 105 * (1 << 23) + 1,
           90 * (1 << 23) + 1, 77 * (1 << 23) + 1, 71 * (1 << 23) + 1]
TGEN = [3, 3, 26, 11, 3, 3]
U32 = np.uint32
M32 = (1 << 32) - 1


def bitrev(i, s):
    r = 0
    while s > 1:
        r = 2 * r | (i & 1)
        i >>= 1
        s >>= 1
    return r


def shoup_const(w, p):
    return (w << 32) // p


def _bitrev_array(s):
    """bitrev(j, s) for j < s (s a power of two)."""
    j = np.arange(s, dtype=np.int64)
    r = np.zeros(s, dtype=np.int64)
    b = s.bit_length() - 1
    for i in range(b):
        r |= ((j >> i) & 1) << (b - 1 - i)
    return r


def _powers(x, s, p):
    """x^j mod p for j < s (numpy, p < 2^30)."""
    out = np.ones(s, dtype=np.uint64)
    j = np.arange(s, dtype=np.int64)
    sq = np.uint64(x % p)
    for i in range(max(1, s.bit_length())):
        sel = ((j >> i) & 1) == 1
        out[sel] = out[sel] * sq % np.uint64(p)
        sq = sq * sq % np.uint64(p)
    return out


def tables(ln, k, domain_q):
    """(w, ws), and for domain R (wi, wis) = -w^-1, at positions s + bitrev(j, s)."""
    p, g = TPRIMES[k], TGEN[k]
    n = 1 << ln
    w = np.zeros(n // 2, dtype=np.uint64)
    wi = np.zeros(n // 2, dtype=np.uint64)
    lvl = ln - 1
    s = n // 4
    while s >= 1:
        rho = pow(g, (p - 1) >> lvl, p)
        rhoi = pow(rho, p - 2, p)
        t0 = pow(g, (p - 1) >> (lvl + 1), p) if domain_q else 1
        pos = s + _bitrev_array(s)
        w[pos] = _powers(rho, s, p) * np.uint64(t0) % np.uint64(p)
        wi[pos] = (np.uint64(p) - _powers(rhoi, s, p)) % np.uint64(p)
        s //= 2
        lvl -= 1
    ws = (w << np.uint64(32)) // np.uint64(p)
    wis = (wi << np.uint64(32)) // np.uint64(p)
    if domain_q:
        return w, ws, None, None
    return w, ws, wi, wis


def _u(x):
    return (np.asarray(x, dtype=np.uint64) & np.uint64(M32))


def shoup(x, w, ws, p):
    x = _u(x)
    q = (x * _u(ws)) >> np.uint64(32)
    return _u(x * _u(w) - q * np.uint64(p))


def redc(t, p, add=1):
    """t 2^-32 mod p of a 64-bit sum: its high word less that of m p, plus `add` p."""
    pinv = pow(p, -1, 1 << 32)
    t = np.asarray(t, dtype=np.uint64)
    lo, hi = t & np.uint64(M32), t >> np.uint64(32)
    m = _u(lo * np.uint64(pinv))
    return _u(hi - ((m * np.uint64(p)) >> np.uint64(32)) + np.uint64(add * p))


def red2(x, p):
    x = _u(x)
    y = _u(x - np.uint64(2 * p))
    return np.minimum(x, y)


def exact_limbs(exact):
    """Three 32-bit limbs (two's complement, 96 bits) of python-int exact values."""
    d = [int(v) & ((1 << 96) - 1) for v in exact]
    d0 = np.array([x & M32 for x in d], dtype=np.uint64)
    d1 = np.array([(x >> 32) & M32 for x in d], dtype=np.uint64)
    d2 = np.array([(x >> 64) & M32 for x in d], dtype=np.uint64)
    return d0, d1, d2


def encode_weights(k, s=1):
    """Weights of the three limbs for image factor s (encode_weights of the engine),
    and whether they are in the encoder's range."""
    p = TPRIMES[k]
    w = [s * pow(2, 32 * (j + 1), p) % p for j in range(3)]
    return w, 2 * w[0] + 2 * w[1] + w[2] <= 4 * p


def encode(exact, k, limbs=None, s=1):
    """Residues in (0, 4p) of s times exact values (python ints, 96 bits), as the column pass."""
    p = TPRIMES[k]
    d0, d1, d2 = exact_limbs(exact) if limbs is None else limbs
    w, ok = encode_weights(k, s)
    assert ok
    top = np.where(d2 >> np.uint64(31) != 0, d2 | np.uint64(M32 << 32), d2)   # sign-extended
    return redc(d0 * np.uint64(w[0]) + d1 * np.uint64(w[1]) + top * np.uint64(w[2]), p, 2)


def forward(x, ln, k, domain_q, reduce_out=False):
    """All ln-1 forward levels (index bit ln-1-l at level l), lazy [0, 4p)."""
    p = TPRIMES[k]
    w, ws, _, _ = tables(ln, k, domain_q)
    x = _u(x).copy()
    n = 1 << ln
    for l in range(ln - 1):
        half = n >> (l + 1)
        i = np.arange(n)
        i0 = i[(i & half) == 0]
        i1 = i0 + half
        j = i0 >> (ln - l)
        tw, tws = w[(1 << l) + j], ws[(1 << l) + j]
        a = red2(x[i0], p)
        t = shoup(x[i1], tw, tws, p)
        x[i0] = _u(a + t)
        x[i1] = _u(a - t + np.uint64(2 * p))
    return red2(x, p) if reduce_out else x


def poly_product(x0, x1, y0, y1, mul, cm, p):
    """(x0 + x1 X)(y0 + y1 X) 2^-32 mod (X^2 - c), cm = c 2^32 mod p; words in [0, 2p)."""
    x0, x1, y0, y1, cm = _u(x0), _u(x1), _u(y0), _u(y1), _u(cm)
    t = redc(x1 * y1, p)
    r0 = redc(x0 * y0 + t * cm, p)
    r1 = redc(x0 * y1 + x1 * y0 if mul else (x0 + x0) * x1, p)
    return red2(r0, p), red2(r1, p)


def pointwise(x, ln, k, domain_q, y=None):
    """Degree-1 products mod (x^2 -+ c), c = w[n/4 + m/2] (Montgomery, outputs [0, 2p))."""
    p = TPRIMES[k]
    _, ws, _, _ = tables(ln, k, domain_q)
    n = 1 << ln
    m = np.arange(n // 2)
    cm = _u(np.uint64(0) - ws[n // 4 + (m >> 1)] * np.uint64(p))     # w 2^32 mod p from its Shoup quotient
    cm = np.where((m & 1) == 0, cm, np.uint64(p) - cm)
    x0, x1 = red2(x[0::2], p), red2(x[1::2], p)
    y0, y1 = (x0, x1) if y is None else (y[0::2], y[1::2])
    out = np.empty(n, dtype=np.uint64)
    out[0::2], out[1::2] = poly_product(x0, x1, y0, y1, y is not None, cm, p)
    return out


def inverse(x, ln, k, domain_q):
    """All inverse levels, with -w^-1 (R: its table; Q: w at the mirrored position)."""
    p = TPRIMES[k]
    w, ws, wi, wis = tables(ln, k, domain_q)
    x = _u(x).copy()
    n = 1 << ln
    for l in reversed(range(ln - 1)):
        half = n >> (l + 1)
        i = np.arange(n)
        i0 = i[(i & half) == 0]
        i1 = i0 + half
        j = i0 >> (ln - l)
        idx = (1 << l) + j
        if domain_q:
            mi = 3 * (1 << l) - 1 - idx
            v, vs = w[mi], ws[mi]
        else:
            v, vs = wi[idx], wis[idx]
        s = _u(x[i0] + x[i1])
        d = _u(x[i1] - x[i0] + np.uint64(2 * p))
        x[i0] = red2(s, p)
        x[i1] = shoup(d, v, vs, p)
    return x


def _sqrt(x, p):
    """A square root of the square x mod p (Tonelli-Shanks, as the engine)."""
    q, m = p - 1, 0
    while q % 2 == 0:
        q, m = q // 2, m + 1
    g = 2
    while pow(g, (p - 1) // 2, p) == 1:
        g += 1
    c, t, r = pow(g, q, p), pow(x, q, p), pow(x, (q + 1) // 2, p)
    while t != 1:
        i, y = 0, t
        while y != 1:
            i, y = i + 1, y * y % p
        b = pow(c, 1 << (m - i - 1), p)
        m, c = i, b * b % p
        t, r = t * c % p, r * b % p
    return r


class Consts:
    """The class's image factors and CRT constants (build_consts of the engine)."""

    def __init__(self, ln, K):
        KP, M30 = K + 1, (1 << 30) - 1
        M = 1
        for p in TPRIMES[:KP]:
            M *= p

        def columns(v):
            c = [(v >> (30 * j)) & M30 for j in range(K - 1)] + [(v >> (30 * (K - 1))) & M32]
            return c, v >> (30 * (K - 1) + 32)
        self.K, self.M, self.s, self.e, self.mk, self.mkh = K, M, [], [], [], []
        total = 0
        for k in range(KP):
            p = TPRIMES[k]
            cw = pow((1 << ln) // 2, -1, p) * ((1 << 32) % p) % p * pow(M // p % p, -1, p) % p
            e = 1
            while pow(cw * pow(e, -1, p) % p, (p - 1) // 2, p) != 1:
                e += 1
            s = _sqrt(cw * pow(e, -1, p) % p, p)
            self.s.append(s if encode_weights(k, s)[1] else p - s)
            assert encode_weights(k, self.s[k])[1]
            self.e.append(e)
            c, h = columns(M // p * e)
            assert h == 0 or (K == 4 and k == 3)
            self.mk.append(c)
            self.mkh.append(h)
            total += M // p * e * 2 * p
        assert (total >> (30 * (K - 1))).bit_length() <= 64
        self.tsh = 0
        while True:
            self.tsh += 1
            t = (1 << (64 + 30 * (K - 1) + self.tsh)) // M
            if t.bit_length() >= 31:
                break
        self.tinv = t
        assert t.bit_length() <= 32
        self.negm, self.negmh = columns(-M % (1 << (32 * K)))


def crt_limbs(c, y):
    """The engine's crt: K limbs of V from the K+1 lazy CRT coordinates."""
    L, u = c.K, np.uint64
    y = [_u(v) for v in y]
    col = []
    for j in range(L):
        a = y[0] * u(c.mk[0][j])
        for k in range(1, L + 1):
            a = a + y[k] * u(c.mk[k][j])
        col.append(a)
    if L == 4:
        col[L - 1] = col[L - 1] + (_u(y[3] * u(c.mkh[3])) << u(32))
    hi = _u((col[L - 1] + (col[L - 2] >> u(30))) >> u(32))
    t = (((hi * u(c.tinv)) >> u(32)) + u(1 << (c.tsh - 1))) >> u(c.tsh)
    for j in range(L):
        col[j] = col[j] + t * u(c.negm[j])
    col[L - 1] = col[L - 1] + (_u(t * u(c.negmh)) << u(32))
    for j in range(1, L):
        col[j] = col[j] + (col[j - 1] >> u(30))
    limbs = []
    for i in range(L - 1):
        pair = (_u(col[i]) << u(2) & u(M32)) | (_u(col[i + 1]) << u(32))
        limbs.append(_u(pair >> u(2 + 2 * i)))
    limbs.append(_u(col[L - 1] >> u(2 * (L - 1))))
    return limbs


def crt(res, ln, K):
    """Exact signed values from the K+1 planes of inverse outputs (each [0, 2p))."""
    limbs = crt_limbs(Consts(ln, K), res)
    out = []
    for i in range(len(limbs[0])):
        v = sum(int(l[i]) << (32 * j) for j, l in enumerate(limbs))
        out.append(v - (1 << (32 * K)) if v >> (32 * K - 1) else v)
    return out


def product(xe, ye, ln, K, domain_q):
    """Exact coefficients of x*y mod (x^n -+ 1) (ye None: x^2) through the model."""
    res, c = [], Consts(ln, K)
    for k in range(K + 1):
        fx = forward(encode(xe, k, s=c.s[k]), ln, k, domain_q)
        fy = None if ye is None else forward(encode(ye, k, s=c.s[k]), ln, k, domain_q, reduce_out=True)
        res.append(inverse(pointwise(fx, ln, k, domain_q, fy), ln, k, domain_q))
    return crt(res, ln, K)


def exact_product(xe, ye, ln, domain_q):
    """Cyclic (R) or negacyclic (Q) convolution with python ints."""
    n = 1 << ln
    ye = xe if ye is None else ye
    out = [0] * n
    for i in range(n):
        xi = int(xe[i])
        if xi == 0:
            continue
        for j in range(n):
            t = i + j
            if t >= n:
                t -= n
                out[t] += -xi * int(ye[j]) if domain_q else xi * int(ye[j])
            else:
                out[t] += xi * int(ye[j])
    return out
