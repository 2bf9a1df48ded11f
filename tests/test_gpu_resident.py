"""Short transforms in one launch per run (resident.cu) against the passes:
the same handle's registers, word for word, for every class and length, with
the digit sizes of the parameter rule and small ones (the general digit
moves); batches with resting slots, snapshots and empty slots."""
import numpy as np
import pytest

import annie_b200 as A
from annie_b200.synth import Xoshiro256ss

pytestmark = pytest.mark.gpu

PCK = {2: 1, 3: 2, 4: 2, 5: 4}


def _number(params, seed):
    K, pck, ln, lbase = params
    rng = Xoshiro256ss(seed)
    while True:
        N = rng.random_odd(max(64, (pck * lbase << ln) // 2 - rng.uniform(0, 40)))
        if not A.probe(N, 3, forced=params)[1]:
            return N


def _default_split(t):
    t.set_geometry(t.geometry()[0])        # an explicit split: the passes


@pytest.mark.parametrize("ln", range(6, 13))
@pytest.mark.parametrize("K,lbase", [(2, 14), (3, 20), (4, 27), (5, 17), (2, 3), (3, 9), (4, 15), (5, 7)])
def test_resident_equals_passes(K, lbase, ln):
    params = (K, PCK[K], ln, lbase)
    N = _number(params, 100 * K + ln)
    t, u = (A.Transform(N, 3, params=params) for _ in range(2))
    _default_split(u)
    for x in (t, u):
        x.set1()
        x.copy(1, 0)
        x.square_mul_bits(0x5a5a5a5a5a5a5a5a5b, 70, 3)
        x.square_mul(7)
        x.mul(1, 0)
        x.square_mul(1)
        x.mul(0, 0)
    assert t.launch_count() < u.launch_count()
    for r in (0, 1):
        assert np.array_equal(t.read_register(r), u.read_register(r)), "Reg%d" % r
    assert t.get(0) == u.get(0)


@pytest.mark.parametrize("bits", [2450, 9000, 36000, 60000, 130000, 262144])
def test_resident_batch_equals_passes(bits):
    rng = Xoshiro256ss(bits)
    nums = []
    while len(nums) < 3:
        N = rng.random_odd(bits)
        p, failed = A.probe(N, 3)
        if not failed:
            nums.append(N)
            cls = p
    batches = []
    for passes in (False, True):
        b = A.Batch(cls, capacity=len(nums) + 2, max_steps=12)
        for s, N in enumerate(nums):
            assert not b.load(s + 1, N, 3)             # slot 0 and the last stay empty
            b.slot(s + 1).set1()
            b.slot(s + 1).copy(1, 0)
        if passes:
            b.set_geometry(b.slot(1).geometry()[0])
        m = np.random.default_rng(bits).choice([1, 3, 5], size=(12, len(nums) + 2)).astype(np.uint32)
        m[9:, 1] = 0                                   # rests at the end
        m[4, -2] = 0                                   # and in the middle
        snap = np.zeros(m.shape, dtype=np.uint8)
        snap[7] = 1
        for _ in range(2):
            b.steps(m, snap)
            for s in range(len(nums)):
                b.gl_mul(s + 1)
        batches.append(b)
    for s in range(len(nums)):
        for r in (0, 1):
            assert np.array_equal(batches[0].slot(s + 1).read_register(r), batches[1].slot(s + 1).read_register(r)), "slot %d" % s
