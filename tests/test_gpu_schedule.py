"""Calls that change a handle's or a batch's schedule between squarings: the
registers do not depend on them, and the default path comes back."""
import numpy as np
import pytest

import annie_b200 as A
from annie_b200.synth import Xoshiro256ss, proth
from test_gpu_resident import PCK, _number

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("K,lbase", [(2, 14), (3, 20), (4, 27), (5, 17)])
def test_overlap_switched_between_squarings(K, lbase):
    # 64 steps at once after single steps with the other overlap, and after a
    # profiled step, against single steps
    params = (K, PCK[K], 13, lbase)
    N = _number(params, K)
    bits = 0xb5e3a1c97d2f4816

    def run(t, switch):
        t.set_overlap(True)
        t.set1()
        t.square_mul(3)
        switch(t)
        for i in range(2):
            t.square_mul_bits(bits >> i, 64, 3)
            t.square_mul(1)
        return t.read_register(0)

    def singles(t):
        t.set_overlap(True)
        t.set1()
        t.square_mul(3)
        for i in range(2):
            for s in range(64):
                t.square_mul(3 if (bits >> i >> s) & 1 else 1)
            t.square_mul(1)
        return t.read_register(0)

    t = A.Transform(N, 3, params=params)
    exp = singles(t)
    assert np.array_equal(run(t, lambda t: None), exp)
    assert np.array_equal(run(t, lambda t: t.set_overlap(False)), exp), "overlap off"

    def off_on(t):
        t.set_overlap(False)
        t.square_mul_bits(0, 0, 3)
        t.set_overlap(True)
    assert np.array_equal(run(t, off_on), exp), "off and on"

    def profiled():
        t.set_overlap(False)
        t.set1()
        t.profile_square(3)
        t.square_mul_bits(bits, 64, 3)
        return t.read_register(0)
    got = profiled()
    t.set_overlap(True)
    t.set1()
    t.square_mul(3)
    t.square_mul_bits(bits, 64, 3)
    assert np.array_equal(got, t.read_register(0)), "profiled step"


@pytest.mark.parametrize("overlap", [True, False])
@pytest.mark.parametrize("K,lbase", [(2, 14), (4, 27), (5, 17)])
def test_get_between_squarings(K, lbase, overlap):
    # reading a register, by value or by its words, leaves the next squaring alone
    params = (K, PCK[K], 13, lbase)
    N = _number(params, K + 10)
    t = A.Transform(N, 3, params=params)
    t.set_overlap(overlap)
    t.set1()
    t.copy(1, 0)
    e = 0
    for i, a in enumerate((3, 1, 3, 3, 1)):
        t.square_mul(a)
        e = 2 * e + (a == 3)
        t.get(i % 2)
        t.read_register(0)
    assert t.get(0) == pow(3, e, N)
