"""Numbers whose polynomial has at most three nonzero coefficients (k 2^m + 1):
the product by N without a transform, against the oracle, for every class, in
the resident runs, in the passes at several splits (a thread per word and a
thread per group), in the allocation-free entry point and in batches."""
import numpy as np
import pytest

import annie_b200 as A

from test_gpu_resident import PCK

pytestmark = pytest.mark.gpu


def _numbers(params):
    """N at the edges: k inside one coefficient, across two, at either end of the
    register; one, two and three terms; and a fourth term (dense)."""
    K, pck, ln, lbase = params
    w, n = pck * lbase, 1 << ln
    top = w * n // 2                         # about half of R, as the parameter rule leaves
    forms = []
    for m in (w, w * (n // 4) + w - 1, w * (n // 4) + w // 2, top - 21, top - w - 3):
        for k in range(524287, 524400, 2):
            forms.append((m, [(k, m)]))
    for k in range(3, 60, 2):
        forms.append(("three", [(k, w * 2 + 5), (1, top)]))
        forms.append(("four", [(k, w * 2), (1, w * 5 + 1), (1, top)]))
    done = set()
    for key, terms in forms:
        N = 1 + sum(k << m for k, m in terms)
        if key not in done and N.bit_length() > 60 and not A.probe(N, 3, forced=params)[1]:
            done.add(key)
            yield N


CASES = [(2, 7, 13), (3, 8, 20), (4, 9, 27), (5, 10, 17), (5, 6, 18), (3, 10, 9), (5, 9, 6), (4, 7, 14)]


@pytest.mark.parametrize("K,ln,lbase", CASES)
def test_sparse_n_equals_oracle(oracle_mod, K, ln, lbase):
    params = (K, PCK[K], ln, lbase)
    count = 0
    for N in _numbers(params):
        o = oracle_mod.Oracle(N, 3, params=params)
        t = A.Transform(N, 3, params=params)
        L, count = ln - 1, count + 1
        o.set1(); o.copy(1, 0)
        for a in (3, 1, 3):
            o.square_mul(a)
        o.mul(1, 0)
        exp = [o.read_reg(r) for r in (0, 1)]
        for lb in [None] + [lb for lb in range(4, L) if L - lb <= 6]:
            if lb is not None:
                t.set_geometry(lb)
            t.set1(); t.copy(1, 0)
            t.square_mul_bits(5, 3, 3)
            t.mul(1, 0)
            for r in (0, 1):
                assert np.array_equal(t.read_register(r), exp[r]), "N = %x, Reg%d, split %s" % (N, r, lb)
            assert t.get(0) == o.get(0)
        t.close()
    assert count >= 5


def test_sparse_n_noalloc(oracle_mod):
    import torch
    for params in ((5, 4, 10, 18), (5, 4, 13, 17)):
        K, pck, ln, lbase = params
        for k in range(3, 99, 2):
            N = (k << (pck * lbase << ln) // 2) + 1
            if not A.probe(N, 3, forced=params)[1]:
                break
        t = A.Transform(N, 3, params=params)
        t.set1()
        t.square_mul_bits(3, 2, 3)
        reg = torch.from_numpy(t.read_register(0).view(np.int32)).cuda()
        torch.cuda.synchronize()
        t.square_mul(3)
        t.square_mul_noalloc(reg.data_ptr(), 3)
        t.synchronize()
        assert np.array_equal(reg.cpu().numpy().view(np.uint32), t.read_register(0))


@pytest.mark.parametrize("bits", [100020, 500020])
def test_sparse_and_dense_slots(bits):
    # a batch of sparse N alone (resident, or passes without the product's
    # transform), then with a dense slot beside them (the passes take all slots
    # as dense), and one that fills the GPU
    from annie_b200.synth import Xoshiro256ss, proth
    rng = Xoshiro256ss(bits)

    def number(dense):
        while True:
            N = rng.random_odd(bits) if dense else proth(rng.uniform(1 << 19, 1 << 20) | 1, bits - 20)
            if not A.probe(N, 3)[1]:
                return N

    nums = [number(False), number(False), number(True)]
    singles = [A.Transform(N, 3) for N in nums]
    cap = 40
    b = A.Batch(A.probe(nums[0], 3)[0], capacity=cap, max_steps=5)
    mult = np.zeros((5, cap), dtype=np.uint32)
    for s, t in enumerate(singles):
        t.set1()
        if s < 2:
            assert not b.load(s, nums[s], 3)
            b.slot(s).set1()

    def step(slots):
        m = mult.copy()
        m[:, slots] = np.array([[3], [1], [1], [3], [1]], dtype=np.uint32)
        b.steps(m)
        for s in {min(s, 2) if s < 3 else 0 for s in slots}:
            singles[s].square_mul_bits(0b01001, 5, 3)
        for s in slots:
            assert np.array_equal(b.slot(s).read_register(0), singles[s if s < 3 else 0].read_register(0)), "slot %d" % s

    step([0, 1])
    assert not b.load(2, nums[2], 3)
    b.slot(2).set1()
    step([0, 1, 2])
    b.release(2)
    for s in range(3, cap):
        b.clone(s, 0)
    step([0, 1] + list(range(3, cap)))
