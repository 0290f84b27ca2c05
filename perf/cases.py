"""The work whose speed is measured: evaluator calls as programs make them.

A case names an operation, a ring degree 2^log_n, `k` Q primes and `kl`
special primes of `bits` bits ("60": the largest 60-bit primes q = 1 mod 2^32,
the primes of the benchmark and of the serving loops; "60g": the largest
q = 1 mod 2N; "55": a 63-bit q_0 before 55-bit primes, the layout of the
reference's own sets; "52": 52-bit primes), the transform the evaluation runs
on and, for batches, the number of operations.  Keys and ciphertexts are real:
the device samplers' keys, encryptions of values in the unit disk.

Engines and contexts are kept per parameter set, as a program keeps them;
keys, ciphertexts and result buffers are made anew from every seed.
"""
import math
import random

import numpy as np
import torch

import aoa_b200 as aoa
from aoa_b200 import AOA_COEF, AOA_DGT, AOA_NTT, capi, params

_SCALE_BITS = {"60": 50, "60g": 50, "55": 50, "52": 40}


def listed():
    return [
        # one product at the smallest parameters in use (N = 2^12, 3 x 52-bit): latency and launches
        {"name": "mul_n12", "op": "mul", "log_n": 12, "k": 3, "kl": 4, "bits": "52", "transform": "ntt", "batch": 1},
        # domain changes of a few polynomials of a small ring, both directions
        {"name": "ntt_n12", "op": "ntt", "log_n": 12, "k": 5, "kl": 0, "bits": "52", "transform": "ntt", "batch": 2},
        # one rotation of a small ring on ordinary primes
        {"name": "rotate_n13", "op": "rotate", "log_n": 13, "k": 6, "kl": 7, "bits": "60g", "transform": "ntt",
         "batch": 1, "step": 37},
        # one product of a middle ring on the reference's prime layout (63-bit q_0, 55-bit primes)
        {"name": "mul_n14_ref", "op": "mul", "log_n": 14, "k": 12, "kl": 13, "bits": "55", "transform": "ntt",
         "batch": 1},
        # encode, encrypt, decrypt, decode on the same primes: what a client does
        {"name": "client_n14_ref", "op": "client", "log_n": 14, "k": 12, "kl": 13, "bits": "55", "transform": "ntt",
         "batch": 1},
        # a serving request: plaintext weights, sum of all slots, rescale
        {"name": "score_n15", "op": "score", "log_n": 15, "k": 30, "kl": 31, "bits": "60", "transform": "ntt",
         "batch": 1, "limbs": 17},
        # products of ciphertexts at different levels in one call
        {"name": "mul_mixed_n15", "op": "mul", "log_n": 15, "k": 30, "kl": 31, "bits": "60", "transform": "ntt",
         "batch": 24, "mixed": True},
        # the DGT evaluator, a small batch of an odd limb count
        {"name": "mul_dgt_n15", "op": "mul", "log_n": 15, "k": 15, "kl": 16, "bits": "60", "transform": "dgt",
         "batch": 7},
        # one product at the headline parameters
        {"name": "mul_n16", "op": "mul", "log_n": 16, "k": 30, "kl": 31, "bits": "60", "transform": "ntt",
         "batch": 1},
        # rotations by different steps, a key per step, at different levels
        {"name": "rotate_steps_n16", "op": "rotate", "log_n": 16, "k": 30, "kl": 31, "bits": "60",
         "transform": "ntt", "batch": 12, "mixed": True},
        # the transforms alone, many limbs of the large ring, both directions
        {"name": "ntt_n16", "op": "ntt", "log_n": 16, "k": 30, "kl": 0, "bits": "60", "transform": "ntt",
         "batch": 64},
        # the headline: a batch of products at full level
        {"name": "mul_batch_n16", "op": "mul", "log_n": 16, "k": 30, "kl": 31, "bits": "60", "transform": "ntt",
         "batch": 48},
    ]


def _log_int(rng, lo, hi):
    """A whole number in [lo, hi], spread over its logarithm."""
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo - 0.49), math.log(hi + 0.49)))))))


def draw(rng):
    op = rng.choice(["mul", "mul", "mul", "rotate", "rotate", "ntt", "ntt", "score", "client"])
    log_n = rng.randint(12, 16)
    bits = rng.choice(["60", "60", "60g", "55", "52"])
    k = rng.randint(3, min(30, 6 + 8 * (log_n - 12)))
    c = {"op": op, "log_n": log_n, "k": k, "kl": k + 1, "bits": bits, "transform": "ntt", "batch": 1}
    if op == "mul":
        c["transform"] = rng.choice(["ntt", "ntt", "dgt"])
        c["batch"] = rng.choice([1, 1, _log_int(rng, 2, 40 if c["transform"] == "ntt" else 20)])
        c["mixed"] = rng.random() < 0.5
    elif op == "rotate":
        c["batch"] = rng.choice([1, _log_int(rng, 2, 12)])
        c["mixed"] = rng.random() < 0.5
        c["step"] = rng.randrange(1, 1 << (log_n - 1))
    elif op == "ntt":
        c["kl"] = 0
        c["transform"] = rng.choice(["ntt", "dgt"])
        c["batch"] = _log_int(rng, 2, 60)
    elif op == "score":
        c["limbs"] = rng.randint(3, k)
    return c


def _primes(case):
    n, k = 2 << case["log_n"], case["k"] + case["kl"]
    if case["bits"] == "60":
        return params.ntt_primes(60, 1 << 32, k)
    if case["bits"] == "55":
        return params.ntt_primes(63, n, 1) + params.ntt_primes(55, n, k - 1)
    return params.ntt_primes(int(case["bits"].rstrip("g")), n, k)


_CONTEXTS = {}


def _context(case):
    """The engine and context of the case's parameters."""
    key = tuple(case[x] for x in ("log_n", "k", "kl", "bits", "transform"))
    if key not in _CONTEXTS:
        p = _primes(case)
        engine = aoa.Engine(case["log_n"], p[:case["k"]], p[case["k"]:], scale_bits=_SCALE_BITS[case["bits"]])
        ctx = aoa.Context(engine)
        if case["transform"] == "dgt":
            ctx.set_transform(AOA_DGT)
        _CONTEXTS[key] = ctx
    return _CONTEXTS[key]


class _Words:
    """The live limbs of a device buffer, as the array interface describes them (keeps the buffer's owner)."""

    def __init__(self, owner, ptr, shape, strides):
        self.owner = owner
        self.__cuda_array_interface__ = {"shape": tuple(shape), "strides": tuple(strides), "typestr": "<i8",
                                         "data": (int(ptr), False), "version": 3}


def _tensor(owner, ptr, shape, strides):
    return torch.as_tensor(_Words(owner, ptr, shape, strides), device="cuda")


def _ct_tensor(ct, limbs):
    E = ct.ctx.engine
    return _tensor(ct, ct.device_ptr.value, (2, limbs, E.N), (E.k * E.N * 8, E.N * 8, 8))


def _limbs(case):
    """Live limbs of each operand: all of them, or spread over 4 .. k (2 .. k below four)."""
    k = case["k"]
    if case["op"] == "score":
        return [case["limbs"]]
    if not case.get("mixed"):
        return [k] * case["batch"]
    r = random.Random(case["batch"])
    return [r.randint(min(4, k - 1), k) for _ in range(case["batch"])]


def _steps(case):
    """The rotation of each operation: the case's, or for a batch every power of two in turn."""
    if case["batch"] == 1:
        return [case.get("step", 1)]
    return [1 << (i % (case["log_n"] - 1)) for i in range(case["batch"])]


def _values(rng, n):
    """n complex values in the unit disk."""
    return np.sqrt(rng.random(n)) * np.exp(2j * np.pi * rng.random(n))


def prepare(case, seed):
    ctx = _context(case)
    E = ctx.engine
    op = case["op"]
    slots = E.N // 2
    rng = np.random.default_rng(seed)
    if op == "ntt":
        shape = (case["batch"], E.k, E.N)
        q = np.array(E.q_primes, dtype=np.int64)
        g = torch.Generator(device="cuda").manual_seed(seed)
        src, work = [], []
        for _ in range(2):                       # one array for each direction
            d = ctx.alloc(shape)
            t = _tensor(d, d.ptr.value, shape, (E.k * E.N * 8, E.N * 8, 8))
            for l in range(E.k):
                t[:, l] = torch.randint(0, int(q[l]), (case["batch"], E.N), generator=g, device="cuda")
            src.append(d)
            w = ctx.alloc(shape)
            work.append((w, _tensor(w, w.ptr.value, shape, (E.k * E.N * 8, E.N * 8, 8))))
        torch.cuda.synchronize()
        return {"case": case, "ctx": ctx, "src": src, "work": work}
    steps = []
    if op == "rotate":
        steps = _steps(case)
    elif op == "score":
        steps = [1 << j for j in range(E.log_n - 1)]
    secret, keys = aoa.ckks_keygen_sampled(ctx, seed, rotations=sorted(set(steps)))
    s = {"case": case, "ctx": ctx, "secret": secret, "keys": keys, "steps": steps}
    if op == "client":
        s.update(values=_values(rng, slots), ct=aoa.Ciphertext(ctx), seed=seed)
        s["out"] = _ct_tensor(s["ct"], E.k)
        return s
    stream = [1000]

    def encryption(limbs):
        ct = aoa.ckks_encrypt_sampled(ctx, _values(rng, slots), keys["pk"], seed, stream=stream[0])
        stream[0] += 3
        _, sl, scale, domain = ct._get()
        ct.set(limbs - 1, sl, scale, domain)     # a ciphertext that earlier operations have brought down
        return ct

    limbs = _limbs(case)
    s["a"] = [encryption(m) for m in limbs]
    s["c"] = [aoa.Ciphertext(ctx) for _ in limbs]
    if op == "mul":
        s["b"] = [encryption(m) for m in limbs]
        s["out"] = [_ct_tensor(c, m - 1) for c, m in zip(s["c"], limbs)]
    elif op == "rotate":
        s["rtk"] = [keys["rtk"][x] for x in steps]
        s["out"] = [_ct_tensor(c, m) for c, m in zip(s["c"], limbs)]
    else:                                        # score: encoded weights, as the serving loop keeps them
        s["weights"] = aoa.ckks_encode(ctx, _values(rng, slots))[0]
        s["sum"] = aoa.Ciphertext(ctx)
        s["out"] = _ct_tensor(s["sum"], limbs[0] - 2)
    ctx.sync()
    return s


def run(s):
    case, ctx, op = s["case"], s["ctx"], s["case"]["op"]
    if op == "mul":
        evk = s["keys"]["evk"]
        if case["batch"] == 1:
            aoa.ckks_mul(ctx, s["c"][0], s["a"][0], s["b"][0], evk)
        else:
            aoa.ckks_mul_batch(ctx, s["c"], s["a"], s["b"], evk)
        return s["out"]
    if op == "rotate":
        if case["batch"] == 1:
            aoa.ckks_rotate_left(ctx, s["c"][0], s["a"][0], s["steps"][0], s["rtk"][0])
        else:
            aoa.ckks_rotate_batch_steps(ctx, s["c"], s["a"], s["steps"], s["rtk"])
        return s["out"]
    if op == "ntt":
        lib = capi.load()
        for d, (w, _) in zip(s["src"], s["work"]):   # the transforms are in place: the arrays are kept
            capi.check(lib.aoa_memcpy_d2d(ctx.handle, w.ptr, d.ptr, d.nbytes))
        fwd, inv = (ctx.ntt_fwd, ctx.ntt_inv) if case["transform"] == "ntt" else (ctx.dgt_fwd, ctx.dgt_inv)
        fwd(s["work"][0][0], case["batch"], 0, case["k"])
        inv(s["work"][1][0], case["batch"], 0, case["k"])
        return [t for _, t in s["work"]]
    if op == "score":
        scale = 1 << ctx.engine.scale_bits
        aoa.ckks_mul_pt(ctx, s["c"][0], s["a"][0], s["weights"], scale, rescale=True)
        aoa.ckks_sumslots(ctx, s["sum"], s["c"][0], s["keys"]["rtk"])
        aoa.ckks_rescale(ctx, s["sum"])
        return s["out"]
    aoa.ckks_encrypt_sampled(ctx, s["values"], s["keys"]["pk"], s["seed"], stream=1000, out=s["ct"])
    return {"decoded": aoa.ckks_decrypt(ctx, s["ct"], s["secret"]), "ct": s["out"]}


def work(case):
    """Every operand, key and encoded polynomial read once, every result written once."""
    limb = 8 << case["log_n"]
    k, kl, op = case["k"], case["kl"], case["op"]
    if op == "ntt":
        return {"bytes": 2 * 2 * case["batch"] * k * limb, "flops": 0}
    if op == "client":                           # values, public key, secret; the ciphertext out and in
        return {"bytes": (2 * k + k + 2 * k + 2 * k) * limb + 2 * limb, "flops": 0}
    limbs = _limbs(case)
    if op == "score":
        m = limbs[0]
        return {"bytes": (3 * m + (case["log_n"] - 1) * 2 * (m - 1 + kl) + 2 * (m - 2)) * limb, "flops": 0}
    if op == "mul":
        key = 2 * (max(limbs) + kl)
        return {"bytes": (key + sum(4 * m + 2 * (m - 1) for m in limbs)) * limb, "flops": 0}
    top = {}
    for step, m in zip(_steps(case), limbs):
        top[step] = max(top.get(step, 0), m)
    return {"bytes": (sum(2 * (m + kl) for m in top.values()) + sum(4 * m for m in limbs)) * limb, "flops": 0}


def tolerance(case):
    """Residues are whole numbers with one right value.  Decoded values follow from them
    by a 64-bit floating transform of log2 N stages."""
    return {"rel": 1e-12, "max": 1e-10} if case["op"] == "client" else "exact"


def exact(case, seed):
    """The values that a client encrypted: decryption returns them up to the encryption's noise, the
    same draws on every side.  Residues are compared as whole numbers."""
    if case["op"] != "client":
        return None
    return {"decoded": _values(np.random.default_rng(seed), 1 << (case["log_n"] - 1)), "ct": None}
