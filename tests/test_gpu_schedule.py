"""Calls that change a handle's or a batch's schedule between squarings: the
registers do not depend on them, and the default path comes back."""
import time

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


@pytest.mark.parametrize("bits", [2450, 60000, 262144])
def test_default_split_restores_resident_runs(bits):
    rng = Xoshiro256ss(bits)
    N = rng.random_odd(bits)
    while A.probe(N, 3)[1]:
        N = rng.random_odd(bits)
    t = A.Transform(N, 3)
    split = t.geometry()

    def launches(f):
        l0 = t.launch_count()
        f()
        return t.launch_count() - l0

    def step():
        t.square_mul_bits(5, 16, 3)
    t.set1()
    assert launches(step) == 1
    t.set_geometry(split[0])
    passes = launches(step)
    assert passes > 1
    t.set_geometry(0)
    assert t.geometry() == split and launches(step) == 1
    t.set1()
    for _ in range(3):
        step()
    exp = t.read_register(0)

    b = A.Batch((t.K, t.pck, t.ln, t.lbase), capacity=2, max_steps=16)
    assert not b.load(0, N, 3)
    b.slot(0).set1()
    m = np.array([[3 if (5 >> i) & 1 else 1, 0] for i in range(16)], dtype=np.uint32)
    counts = []
    for lb in (None, split[0], 0):
        if lb is not None:
            b.set_geometry(lb)
        l0 = b.launch_count()
        b.steps(m)
        counts.append(b.launch_count() - l0)
    assert counts[0] == counts[2] == 1 and counts[1] > 1
    assert np.array_equal(b.slot(0).read_register(0), exp)
    # the slot's own view squares resident again too
    v = b.slot(0)
    l0 = v.launch_count()
    v.square_mul_bits(5, 16, 3)
    assert v.launch_count() - l0 == 1


@pytest.mark.parametrize("bits,resident", [(20000, True), (262144, True), (400000, False)])
def test_profile_times_the_launches_of_a_squaring(bits, resident):
    rng = Xoshiro256ss(bits + 1)
    N = rng.random_odd(bits)
    while A.probe(N, 3)[1]:
        N = rng.random_odd(bits)
    t, u = A.Transform(N, 3), A.Transform(N, 3)
    for x in (t, u):
        x.set1()
        x.square_mul(3)
    ms = t.profile_square(3)
    l0 = u.launch_count()
    u.square_mul(3)
    assert len(ms) == u.launch_count() - l0 and (len(ms) == 1) == resident
    assert all(0.0 < x < 5.0 for x in ms)
    assert np.array_equal(t.read_register(0), u.read_register(0))
    # a handle that was given a split is profiled by its passes
    t.set_geometry(t.geometry()[0])
    assert len(t.profile_square(3)) > 1


def _numbers(bits):
    """A dense N and a sparse one (k 2^m + 1) of one class."""
    rng = Xoshiro256ss(bits)

    def number(draw):
        while True:
            N = draw()
            if not A.probe(N, 3)[1]:
                return N
    dense = number(lambda: rng.random_odd(bits))
    sparse = number(lambda: proth(rng.uniform(1 << 19, 1 << 20) | 1, bits - 20))
    assert A.probe(dense, 3)[0][:3] == A.probe(sparse, 3)[0][:3]
    return dense, sparse


def test_remembered_split_is_that_of_the_schedule():
    # a split tuned with sparse N (a squaring without the last product's
    # transform) is not taken for dense N, and the reverse
    cap, steps = 7, 4
    numbers = _numbers(500020)
    tuned = []
    for i in (1, 0, 1, 0):
        b = A.Batch(A.probe(numbers[i], 3)[0], capacity=cap, max_steps=steps)
        assert not b.load(0, numbers[i], 3)
        b.slot(0).set1()
        lb = b.autotune(0, steps)
        assert lb == b.slot(0).geometry()[0]
        tuned.append((b.launch_count() > 0, lb))
        b.close()
    assert [x[0] for x in tuned] == [True, True, False, False]
    assert tuned[0][1] == tuned[2][1] and tuned[1][1] == tuned[3][1]


def test_schedules_of_a_batch_keep_their_graphs():
    # a dense slot that comes and goes changes the batch's schedule; each
    # schedule's graph is captured once
    dense, sparse = _numbers(500020)
    steps = 64
    b = A.Batch(A.probe(sparse, 3)[0], capacity=2, max_steps=steps)
    t = A.Transform(sparse, 3)
    t.set1()
    assert not b.load(0, sparse, 3)
    b.slot(0).set1()
    m = np.zeros((steps, 2), dtype=np.uint32)
    m[:, 0] = [3 if i % 3 == 0 else 1 for i in range(steps)]
    bits = sum(1 << i for i in range(0, steps, 3))
    cost = []
    for i in range(16):
        if i % 2:
            assert not b.load(1, dense, 3)
        else:
            b.release(1)
        b.synchronize()
        t0 = time.perf_counter()
        b.steps(m)
        cost.append(time.perf_counter() - t0)
        b.synchronize()
        t.square_mul_bits(bits, steps, 3)
    assert np.array_equal(b.slot(0).read_register(0), t.read_register(0))
    # host time of a chunk: capturing 64 squarings against a launch
    assert min(cost[2:]) < 0.5 * min(cost[:2]), cost
    assert sorted(cost[2:])[len(cost[2:]) // 2] < 0.5 * min(cost[:2]), cost
