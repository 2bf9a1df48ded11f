"""The column pass with a thread per tile word (launches that do not fill the
GPU, up to 16 rows) against the one with a thread per group of 4 columns."""
import numpy as np
import pytest

import annie_b200 as A

from test_gpu_resident import PCK, _number

pytestmark = pytest.mark.gpu


def _run(t):
    t.set1()
    t.copy(1, 0)
    t.square_mul_bits(0x2d, 6, 3)
    t.mul(1, 0)
    return [t.read_register(r) for r in (0, 1)]


@pytest.mark.parametrize("row_levels", [8, 9, 10, 11])
@pytest.mark.parametrize("K,lbase", [(2, 9), (3, 20), (4, 27), (5, 17), (4, 14), (5, 5)])
def test_wide_columns_equal_grouped(K, lbase, row_levels):
    # 16, 8, 4 and 2 rows of words against 64 rows
    params = (K, PCK[K], 13, lbase)
    t = A.Transform(_number(params, 7 * K + lbase), 3, params=params)
    t.set_geometry(6)
    grouped = _run(t)
    for overlap in (True, False):
        t.set_overlap(overlap)
        t.set_geometry(row_levels)
        for got, exp in zip(_run(t), grouped):
            assert np.array_equal(got, exp)


@pytest.mark.parametrize("bits,row_levels", [(400000, 10), (400000, 8), (900000, 10)])
def test_wide_columns_equal_large_batch(bits, row_levels):
    # a batch whose launches fill the GPU: grouped at every number of rows
    from annie_b200.synth import Xoshiro256ss
    rng = Xoshiro256ss(bits)
    N = rng.random_odd(bits)
    while A.probe(N, 3)[1]:
        N = rng.random_odd(bits)
    t = A.Transform(N, 3)
    b = A.Batch((t.K, t.pck, t.ln, t.lbase), capacity=40, max_steps=6)
    assert not b.load(0, N, 3)
    b.slot(0).set1()
    for s in range(1, 40):
        b.clone(s, 0)
    b.set_geometry(row_levels)
    t.set_geometry(row_levels)
    t.set1()
    t.square_mul_bits(0x2d, 6, 3)
    b.steps(np.repeat(np.array([[3 if (0x2d >> i) & 1 else 1] for i in range(6)], dtype=np.uint32), 40, axis=1))
    for s in (0, 39):
        assert np.array_equal(b.slot(s).read_register(0), t.read_register(0))
