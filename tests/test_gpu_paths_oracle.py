"""Each path of a squaring against the oracle, with dense and sparse N: resident
runs of every class and length, runs of 64 squarings from the captured graph of a
single handle (two streams and one), the column pass by a thread per word and by a
thread per group."""
import numpy as np
import pytest

import annie_b200 as A
from test_gpu_resident import PCK, _number

pytestmark = pytest.mark.gpu


def _sparse(params):
    K, pck, ln, lbase = params
    for k in range(524287, 524500, 2):
        N = (k << (pck * lbase << ln) // 2) + 1
        if not A.probe(N, 3, forced=params)[1]:
            return N


def _pair(oracle_mod, params, sparse):
    N = _sparse(params) if sparse else _number(params, 17 * params[0] + params[2])
    return A.Transform(N, 3, params=params), oracle_mod.Oracle(N, 3, params=params)


def _same(t, o, what):
    for r in (0, 1):
        assert np.array_equal(t.read_register(r), o.read_reg(r)), "%s: Reg%d" % (what, r)


@pytest.mark.parametrize("ln", range(6, 13))
@pytest.mark.parametrize("K,lbase", [(2, 14), (3, 20), (4, 27), (5, 17), (3, 9), (4, 15), (5, 13)])
def test_resident_runs(oracle_mod, K, lbase, ln):
    t, o = _pair(oracle_mod, (K, PCK[K], ln, lbase), False)
    bits, count = 0x1b5e3a1c97d2f48165a, 66                 # a launch of 64 and one of 2
    t.set1(); o.set1()
    t.copy(1, 0); o.copy(1, 0)
    l0 = t.launch_count()
    t.square_mul_bits(bits, count, 3)
    assert t.launch_count() - l0 == 2
    for i in range(count):
        o.square_mul(3 if (bits >> i) & 1 else 1)
    t.mul(1, 0); o.mul(1, 0)
    _same(t, o, "run and product")
    t.square_mul(5); o.square_mul(5)
    t.mul(0, 0); o.mul(0, 0)
    _same(t, o, "single calls")
    assert t.get(0) == o.get(0)


@pytest.mark.parametrize("sparse", [False, True])
@pytest.mark.parametrize("K,lbase,ln", [(2, 13, 13), (3, 20, 13), (4, 27, 13), (5, 17, 13), (4, 15, 14), (5, 17, 14)])
def test_graph_runs(oracle_mod, K, lbase, ln, sparse):
    t, o = _pair(oracle_mod, (K, PCK[K], ln, lbase), sparse)
    t.set1(); o.set1()
    t.copy(1, 0); o.copy(1, 0)
    rng = np.random.default_rng(K * ln)
    for overlap in (True, False):
        t.set_overlap(overlap)
        count = 2 * 64 + 5
        bits = int.from_bytes(rng.bytes(24), "little") & ((1 << count) - 1)
        l0 = t.launch_count()
        t.square_mul_bits(bits, count, 3)
        assert t.launch_count() - l0 > 2 * 64 * 4
        for i in range(count):
            o.square_mul(3 if (bits >> i) & 1 else 1)
        t.mul(1, 0); o.mul(1, 0)
        _same(t, o, "overlap %s" % overlap)
    assert t.get(1) == o.get(1)


@pytest.mark.parametrize("K,lbase", [(2, 13), (3, 20), (4, 27), (5, 17), (4, 14), (5, 12)])
def test_column_pass_by_word_and_by_group(oracle_mod, K, lbase):
    # 2, 8, 16 rows: a thread per word; 32 and 64 rows: a thread per group
    t, o = _pair(oracle_mod, (K, PCK[K], 13, lbase), False)
    t.set1(); o.set1()
    t.copy(1, 0); o.copy(1, 0)
    for row_levels in (11, 9, 8, 7, 6):
        t.set_geometry(row_levels)
        for a in (3, 1):
            t.square_mul(a); o.square_mul(a)
        t.mul(1, 0); o.mul(1, 0)
        _same(t, o, "%d row levels" % row_levels)


def test_column_pass_by_group_at_few_rows(oracle_mod):
    # a batch that fills the GPU: a thread per group at 2, 8 and 16 rows
    from annie_b200.synth import Xoshiro256ss
    rng = Xoshiro256ss(5)
    while True:
        N = rng.random_odd(400000)
        params, failed = A.probe(N, 3)
        if not failed:
            break
    cap = 40
    o = oracle_mod.Oracle(N, 3, params=params)
    b = A.Batch(params, capacity=cap, max_steps=4)
    assert not b.load(0, N, 3)
    b.slot(0).set1()
    o.set1()
    for s in range(1, cap):
        b.clone(s, 0)
    m = np.repeat(np.array([[3], [1], [3], [1]], dtype=np.uint32), cap, axis=1)
    for row_levels in (11, 9, 8):
        b.set_geometry(row_levels)
        b.steps(m)
        for a in (3, 1, 3, 1):
            o.square_mul(a)
        for s in (0, cap - 1):
            assert np.array_equal(b.slot(s).read_register(0), o.read_reg(0)), "%d row levels, slot %d" % (row_levels, s)
