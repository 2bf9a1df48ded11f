"""The work that users of the engine have it do, as measurable cases.

A case is a dict of plain values; `prepare` builds what a program holds before
the call (numbers, transforms, batches, page-locked checkpoint buffers), `run`
makes one pass through the public entry points.  Kinds:

* block   what a test does between two looks at it: resume from a checkpoint
          in page-locked memory, `steps` squarings of the exponent's bits, the
          Gerbicz-Li product, checkpoint back out.
* dropin  the transform interface as a host loop drives it: one square_mul
          call per bit, the Gerbicz-Li product, and the residue read back.
* single  one allocation-free squaring of a register that the caller owns.
* batch   candidates of one size class squared together: chunks that end with
          the Gerbicz-Li snapshot, every slot's product after each, and every
          slot's checkpoint.
* prp     one whole probable-prime test.
* serve   whole tests of mixed sizes through the continuous-batching runner.
"""
import functools
import math

import numpy as np
import torch

import annie_b200 as A
from annie_b200.synth import Xoshiro256ss, euler_base, proth

# Numbers above this many bits take seconds of host set-up (N^-1 mod R), so a
# program keeps their transform for the whole test; the cases do the same.
KEEP_BITS = 4_000_000
# The shortest numbers: below, the NTT length is under the engine's shortest.
MIN_BITS = 2500
SMALL_PRIMES = [p for p in range(3, 2000) if all(p % q for q in range(2, math.isqrt(p) + 1))]


def listed():
    return [
        # the smallest call: one squaring of a caller's register, 70,000 bits
        # (the size of the package's smoke check)
        {"name": "single_70k", "kind": "single", "form": "odd", "bits": 70000},
        # the smallest tests: a few thousand bits, all launch latency
        {"name": "block_2500", "kind": "block", "form": "odd", "bits": 2500, "steps": 64},
        # the transform interface driven call by call by a C++ host
        {"name": "dropin_60k", "kind": "dropin", "form": "odd", "bits": 60000, "steps": 200},
        # a Proth test of 100,000 bits (a size of the reference vectors)
        {"name": "block_proth_100k", "kind": "block", "form": "proth", "bits": 100020, "steps": 256},
        # the full-test configuration: random odd 262,144-bit N, blocks of 256
        {"name": "block_262k", "kind": "block", "form": "odd", "bits": 262144, "steps": 256},
        # k*2^2000000+1 (20-bit k), its Gerbicz-Li block of 977 squarings
        {"name": "block_proth_2M", "kind": "block", "form": "proth", "bits": 2000020, "steps": 977},
        # between the benchmark's sizes: an odd length, four primes of the reference
        {"name": "block_6M", "kind": "block", "form": "odd", "bits": 6643857, "steps": 256},
        # the headline: random odd 33,219,281-bit N, 512 squarings a checkpoint
        {"name": "block_33M", "kind": "block", "form": "odd", "bits": 33219281, "steps": 512},
        # a size class of the Proth sieve n in [500000, 3000000], 16 at a time
        {"name": "batch_proth_1M", "kind": "batch", "form": "proth", "bits": 1_100_000, "slots": 16, "steps": 64, "chunks": 4},
        # many small candidates of one class
        {"name": "batch_20k", "kind": "batch", "form": "odd", "bits": 20000, "slots": 64, "steps": 80, "chunks": 4},
        # one whole Fermat test, call to verdict
        {"name": "prp_10k", "kind": "prp", "form": "odd", "bits": 10007},
        # whole tests of mixed sizes, half Fermat and half Proth, admitted together
        {"name": "serve_2k_8k", "kind": "serve", "lo": 2500, "hi": 8000, "count": 32},
    ]


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["block", "block", "block", "batch", "batch", "single", "dropin", "prp", "serve"])
    form = rng.choice(["odd", "proth"])
    if kind == "single":
        return {"kind": kind, "form": form, "bits": _log_uniform(rng, MIN_BITS, 2_000_000)}
    if kind == "dropin":
        return {"kind": kind, "form": form, "bits": _log_uniform(rng, MIN_BITS, 1_000_000), "steps": rng.randint(32, 300)}
    if kind == "batch":
        bits = _log_uniform(rng, MIN_BITS, 2_000_000)
        slots = rng.randint(2, max(2, min(64, 24_000_000 // bits)))
        return {"kind": kind, "form": form, "bits": bits, "slots": slots, "steps": rng.choice([32, 64, 100]), "chunks": rng.randint(2, 4)}
    if kind == "prp":
        return {"kind": kind, "form": form, "bits": _log_uniform(rng, MIN_BITS, 14000)}
    if kind == "serve":
        lo = _log_uniform(rng, MIN_BITS, 4000)
        return {"kind": kind, "lo": lo, "hi": lo + rng.randint(500, 5000), "count": rng.randint(4, 40)}
    bits = _log_uniform(rng, MIN_BITS, 33_000_000)
    return {"kind": kind, "form": form, "bits": bits, "steps": rng.randint(48, max(64, min(512, 4_000_000_000 // bits)))}


# ------------------------------------------------------------------ numbers
def _shares_small_factor(N, params):
    """A prime below 2000 divides both N and R = 2^(pck lbase 2^ln) - 1."""
    _, pck, ln, lbase = params
    e = pck * lbase << ln
    return any(pow(2, e, p) == 1 and N % p == 0 for p in SMALL_PRIMES)


def _number(form, bits, rng):
    """(N, base, is Proth): the next draw of the form that the engine can test."""
    while True:
        if form == "proth":
            N = proth(rng.uniform(1 << 19, 1 << 20) | 1, bits - 20)
            a = euler_base(N)
        else:
            N = rng.random_odd(bits)
            a = 3
        if not _shares_small_factor(N, A.probe(N, a, gcd=False)[0]):
            return N, a, form == "proth"


def _transform(form, bits, rng):
    while True:
        N, a, _ = _number(form, bits, rng)
        t = A.Transform(N, a)
        if not t.init_failed():
            return t
        t.close()


@functools.lru_cache(maxsize=4)
def _kept_transform(form, bits):
    return _transform(form, bits, Xoshiro256ss(bits))


def _random_bits(rng, count):
    return rng.random_odd(max(2, count)) & ((1 << count) - 1)


def _fill(t, rng):
    """Registers as in the middle of a test: full-size residues in Reg0 and Reg1."""
    t.set1()
    t.square_mul_bits(_random_bits(rng, 64), 64, t.a)
    t.copy(1, 0)
    t.square_mul_bits(_random_bits(rng, 64), 64, t.a)


def _pinned(t):
    """A page-locked buffer for a checkpoint of t."""
    return torch.empty(t.L.ab_checkpoint_size(t.h) // 4, dtype=torch.int32, pin_memory=True)


def _save(t, buf):
    t.save_checkpoint_into(buf.data_ptr(), 4 * buf.numel())


# ------------------------------------------------------------------ prepare
def prepare(case, seed):
    rng = Xoshiro256ss(seed)
    return _PREPARE[case["kind"]](case, rng)


def _prepare_block(case, rng):
    form, bits = case["form"], case["bits"]
    t = _kept_transform(form, bits) if bits > KEEP_BITS else _transform(form, bits, rng)
    _fill(t, rng)
    ckpt, out = _pinned(t), _pinned(t)
    _save(t, ckpt)
    return {"kind": "block", "t": t, "ckpt": ckpt, "out": out, "steps": case["steps"],
            "bits": _random_bits(rng, case["steps"])}


def _prepare_dropin(case, rng):
    t = _transform(case["form"], case["bits"], rng)
    t.set1()
    bits = _random_bits(rng, case["steps"])
    return {"kind": "dropin", "t": t, "mults": [t.a if (bits >> i) & 1 else 1 for i in range(case["steps"])],
            "nbytes": 8 * ((case["bits"] + 63) // 64)}


def _prepare_single(case, rng):
    t = _transform(case["form"], case["bits"], rng)
    _fill(t, rng)
    reg = torch.from_numpy(t.read_register(0).view(np.int32)).cuda()
    torch.cuda.synchronize()
    return {"kind": "single", "t": t, "reg": reg}


def _prepare_batch(case, rng):
    nums = [_number(case["form"], case["bits"], rng)]
    cls = A.probe(nums[0][0], nums[0][1], gcd=False)[0]
    while len(nums) < case["slots"]:
        # the class's other candidates: up to 10 % shorter
        N = _number(case["form"], int(case["bits"] * (1 - 0.1 * rng.random())), rng)
        if A.probe(N[0], N[1], gcd=False)[0][:3] == cls[:3]:
            nums.append(N)
    steps = case["steps"]
    b = A.Batch(cls, capacity=len(nums), max_steps=steps)
    failed = b.load_many([(i, N, a) for i, (N, a, _) in enumerate(nums)])
    live = [i for i, f in enumerate(failed) if not f]
    slots = [b.slot(i) for i in live]
    for t in slots:
        _fill(t, rng)
    bits = [_random_bits(rng, steps) for _ in nums]
    mult = np.array([[nums[i][1] if (bits[i] >> s) & 1 else 1 for i in range(len(nums))] for s in range(steps)], dtype=np.uint32)
    snap = np.zeros((steps, len(nums)), dtype=np.uint8)
    snap[-1] = 1
    return {"kind": "batch", "b": b, "live": live, "chunks": case["chunks"], "slots": slots, "mult": mult, "snap": snap,
            "out": [_pinned(t) for t in slots]}


def _prepare_prp(case, rng):
    N, a, euler = _number(case["form"], case["bits"], rng)
    return {"kind": "prp", "N": N, "euler": euler, "base": 0 if euler else a}


def _requests(case, rng):
    lo, hi = math.log(case["lo"]), math.log(case["hi"])
    return [_number("proth" if i % 2 else "odd", int(math.exp(lo + (hi - lo) * rng.random())), rng) for i in range(case["count"])]


def _prepare_serve(case, rng):
    return {"kind": "serve", "runner": A.Runner(chunk=32), "reqs": _requests(case, rng)}


_PREPARE = {"block": _prepare_block, "dropin": _prepare_dropin, "single": _prepare_single, "batch": _prepare_batch,
            "prp": _prepare_prp, "serve": _prepare_serve}


# ------------------------------------------------------------------ run
def run(state):
    return _RUN[state["kind"]](state)


def _run_block(s):
    t = s["t"]
    t.read_checkpoint_from(s["ckpt"].data_ptr(), 4 * s["ckpt"].numel())
    t.square_mul_bits(s["bits"], s["steps"], t.a)
    t.mul(1, 0)
    _save(t, s["out"])
    return s["out"]


def _run_dropin(s):
    t = s["t"]
    t.set1()
    t.copy(1, 0)
    for m in s["mults"]:
        t.square_mul(m)
    t.mul(1, 0)
    return [np.frombuffer(t.get(r).to_bytes(s["nbytes"], "little"), dtype=np.int64) for r in (0, 1)]


def _run_single(s):
    t = s["t"]
    t.square_mul_noalloc(s["reg"].data_ptr(), t.a)
    t.synchronize()          # other handles' calls share the scratch
    return s["reg"]


def _run_batch(s):
    b = s["b"]
    for _ in range(s["chunks"]):
        b.steps(s["mult"], s["snap"])
        for i in s["live"]:
            b.gl_mul(i)
    for t, buf in zip(s["slots"], s["out"]):
        _save(t, buf)
    return s["out"]


def _signed64(u):
    return u - (1 << 64) if u >> 63 else u


def _run_prp(s):
    r = A.prp_check(s["N"], euler=s["euler"], base=s["base"])
    return {"is_prp": int(r["is_prp"]), "res64": _signed64(r["res64"]), "status": int(r["status"])}


def _run_serve(s):
    r, done = s["runner"], {}
    for tag, (N, a, euler) in enumerate(s["reqs"]):
        r.submit(N, euler=euler, base=0 if euler else a, tag=tag)
    while len(done) < len(s["reqs"]):
        r.advance()
        done.update(r.poll())
    got = [done[tag] for tag in range(len(s["reqs"]))]
    return {"is_prp": np.array([int(g["is_prp"]) for g in got]), "res64": np.array([_signed64(g["res64"]) for g in got], dtype=np.int64),
            "status": np.array([int(g["status"]) for g in got])}


_RUN = {"block": _run_block, "dropin": _run_dropin, "single": _run_single, "batch": _run_batch, "prp": _run_prp, "serve": _run_serve}


# ------------------------------------------------------------------ what a pass needs
def _class(form, bits):
    """(K, n, levels) of a number of this size."""
    N = proth((1 << 20) - 1, bits - 20) if form == "proth" else (1 << bits) - 1
    K, _, ln, _ = A.probe(N, 3, gcd=False)[0]
    return K, 1 << ln, ln - 1


def _squaring_ops(K, n, levels):
    """32-bit integer operations of one squaring: eight transforms of n words
    mod K primes (a butterfly: one modular product of 3 operations, 3 additive
    ones), four pointwise products, and four carries (K words from K residues:
    K^2 multiply-adds)."""
    return 8 * K * (n // 2) * levels * 6 + 4 * K * n * 10 + 4 * n * 2 * K * K


def work(case):
    kind = case["kind"]
    if kind == "serve":
        mid = math.sqrt(case["lo"] * case["hi"])
        K, n, levels = _class("odd", int(mid))
        return {"bytes": case["count"] * mid / 4, "flops": case["count"] * mid * _squaring_ops(K, n, levels)}
    K, n, levels = _class(case["form"], case["bits"])
    reg, ops = 4 * K * n, _squaring_ops(K, n, levels)
    if kind == "single":
        # the register in and out, the images of N and N^-1
        return {"bytes": 4 * reg, "flops": ops}
    if kind == "prp":
        return {"bytes": case["bits"] / 4, "flops": case["bits"] * ops}
    if kind == "dropin":
        return {"bytes": 2 * reg + case["bits"] / 4, "flops": (case["steps"] + 1) * ops}
    if kind == "batch":
        # per slot: Reg0 and Reg1 in and out, the images of N and N^-1
        return {"bytes": case["slots"] * 6 * reg, "flops": case["slots"] * case["chunks"] * (case["steps"] + 1) * ops}
    return {"bytes": 6 * reg, "flops": (case["steps"] + 1) * ops}


# ------------------------------------------------------------------ exact
def _limbs(x, nbytes):
    return np.frombuffer(x.to_bytes(nbytes, "little"), dtype=np.int64)


def _exact_test(N, a, euler):
    x = pow(a, (N - 1) // 2, N) if euler else pow(a, N - 1, N)
    r = x * x % N if euler else x
    return int(x == (N - 1 if euler else 1)), _signed64(r & ((1 << 64) - 1))


def exact(case, seed):
    """The same numbers by Python integers.  Register words depend on the
    engine's redundant digits, so the kinds that return them have no such value."""
    kind, rng = case["kind"], Xoshiro256ss(seed)
    if kind == "prp":
        prp, res = _exact_test(*_number(case["form"], case["bits"], rng))
        return {"is_prp": prp, "res64": res, "status": 0}
    if kind == "serve":
        got = [_exact_test(*q) for q in _requests(case, rng)]
        return {"is_prp": np.array([g[0] for g in got]), "res64": np.array([g[1] for g in got], dtype=np.int64),
                "status": np.zeros(len(got), dtype=np.int64)}
    if kind == "dropin":
        # the multipliers follow the number in the generator's stream (redraws of
        # a number with a large factor in common with R included)
        while True:
            N, a, _ = _number(case["form"], case["bits"], rng)
            if not A.probe(N, a)[1]:
                break
        bits, e = _random_bits(rng, case["steps"]), 0
        for i in range(case["steps"]):
            e = 2 * e + ((bits >> i) & 1)
        x = pow(a, e, N)
        nbytes = 8 * ((case["bits"] + 63) // 64)
        return [_limbs(x, nbytes), _limbs(x, nbytes)]
    return None
