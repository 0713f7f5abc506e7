"""The work whose speed is measured: products in Z_q[x]/(x^N+1), YASHE multiplies,
transforms, encryption with decryption and mixed batches, each through the public
Python binding of the C library.

Sizes are the library's own: N = 1024 .. 16384, q of 62, 127, 190 and 380 bits (the
serving and batching workloads), single calls, serving-sized batches, odd batches, a
limb count without specialised kernels, and the 4096-pair throughput step. Schedules are
the library's defaults, as a program that never calls the autotuner gets them.
Operands are uniform in [0, q), as ciphertexts and evaluation keys are.
"""
import functools
import math

import numpy as np
import torch

import cuyashe_gb300 as cy
from cuyashe_gb300.api import MixedPlan

DEV = "cuda"


# ---- the cases --------------------------------------------------------------------
def listed():
    return [
        # one small product: what a caller of Polynomial::operator* issues, latency only
        {"name": "mul_n1024_q62_b1", "kind": "mul", "n": 1024, "qbits": 62, "batch": 1},
        # products batched at the size the library is quoted at
        {"name": "mul_n4096_q127_b512", "kind": "mul", "n": 4096, "qbits": 127, "batch": 512},
        # an odd batch of a modulus of four limbs, which has no kernels of its own
        {"name": "mul_n8192_q250_b37", "kind": "mul", "n": 8192, "qbits": 250, "batch": 37},
        # one ciphertext pair, relinearised: the unbatched homomorphic multiply
        {"name": "he_n4096_q127_b1", "kind": "he", "n": 4096, "qbits": 127, "t": 1024, "relin": True, "batch": 1},
        # batches as the serving loop forms them, smallest and middle class
        {"name": "he_n2048_q62_b96", "kind": "he", "n": 2048, "qbits": 62, "t": 17, "relin": True, "batch": 96},
        {"name": "he_n8192_q190_b33", "kind": "he", "n": 8192, "qbits": 190, "t": 65537, "relin": True, "batch": 33},
        # the throughput step: 4096 pairs
        {"name": "he_n4096_q127_b4096", "kind": "he", "n": 4096, "qbits": 127, "t": 1024, "relin": True, "batch": 4096},
        # the deep level: twelve 32-bit words, 64 pairs
        {"name": "he_n16384_q380_b64", "kind": "he", "n": 16384, "qbits": 380, "t": 65537, "relin": True, "batch": 64},
        # standalone transforms of residue vectors, both directions, more than L2 holds
        {"name": "ntt_fwd_n4096_q127_b2048", "kind": "ntt", "n": 4096, "qbits": 127, "inverse": False, "batch": 2048},
        {"name": "ntt_inv_n8192_q190_b509", "kind": "ntt", "n": 8192, "qbits": 190, "inverse": True, "batch": 509},
        # a client's encryption of 256 plaintexts and their decryption
        {"name": "crypt_n4096_q127_b256", "kind": "crypt", "n": 4096, "qbits": 127, "t": 1024, "batch": 256},
        # 192 relinearised multiplies of three classes in one prepared launch
        {"name": "mixed_he_b192", "kind": "mixed", "per_class": 64},
    ]


def draw(rng):
    """A case of the same ranges: N a power of two, any size of q, batches over their logarithm."""
    while True:
        kind = rng.choice(["mul", "mul", "he", "he", "he", "ntt", "crypt"])
        n = 1 << rng.randint(10, 14)
        qbits = int(round(math.exp(rng.uniform(math.log(48), math.log(380)))))
        batch = int(round(math.exp(rng.uniform(0.0, math.log(2048)))))
        case = {"kind": kind, "n": n, "qbits": qbits, "batch": batch}
        if kind == "he":
            case["t"] = rng.choice([17, 1024, 65537])
            case["relin"] = rng.random() < 0.75
        elif kind == "ntt":
            case["inverse"] = rng.random() < 0.5
        elif kind == "crypt":
            case["t"] = rng.choice([17, 1024])
            case["n"], case["qbits"] = min(n, 8192), min(qbits, 190)
        most = 0.25 * _transforms({"kind": "he", "n": 4096, "qbits": 127, "relin": True, "batch": 4096}) * 4096 * 12
        if _transforms(case) * case["n"] * math.log2(case["n"]) <= most:
            return case


# ---- moduli and inputs ------------------------------------------------------------
def _is_prime(x):
    d, r = x - 1, 0
    while d % 2 == 0:
        d, r = d // 2, r + 1
    for a in (2, 3, 5, 7, 11, 13, 17, 19, 23, 29, 31, 37):
        y = pow(a, d, x)
        if y in (1, x - 1):
            continue
        for _ in range(r - 1):
            y = y * y % x
            if y == x - 1:
                break
        else:
            return False
    return True


@functools.lru_cache(maxsize=None)
def modulus(bits):
    """The largest prime below 2^bits that is 1 modulo 2^16."""
    q = ((2**bits - 2) >> 16 << 16) + 1
    while not _is_prime(q):
        q -= 1 << 16
    return q


def _generator(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(int(seed) + 1)
    return g


def _uniform(g, count, n, q):
    """[count][n][limbs] words of values uniform below the top limb of q times 2^(64 (limbs - 1))."""
    limbs = (q.bit_length() + 63) // 64
    x = torch.randint(-(2**63), 2**63 - 1, (count, n, limbs), generator=g, device=DEV, dtype=torch.int64)
    top = q >> (64 * (limbs - 1))
    if top < 2**63:
        x[..., limbs - 1] = torch.randint(0, max(1, top), (count, n), generator=g, device=DEV, dtype=torch.int64)
    else:
        x[..., limbs - 1] &= 2**63 - 1  # below half of q
    return x


def _host(x):
    return x.cpu().numpy().view(np.uint64)


MIXED = ((2048, 62, 17), (4096, 127, 1024), (8192, 190, 65537))


def _inputs(case, seed):
    """The tensors of a case (for "mixed": a list of them, one per class), from the seed alone."""
    g = _generator(seed)

    def pairs(n, bits, batch, keys):
        q = modulus(bits)
        d = {"key": _uniform(g, 2 + math.ceil(bits / 32), n, q)} if keys else {}  # f, h and the evaluation key
        return dict(d, a=_uniform(g, batch, n, q), b=_uniform(g, batch, n, q))

    kind = case["kind"]
    if kind == "mixed":
        return [pairs(n, bits, case["per_class"], True) for n, bits, _ in MIXED]
    n, bits, batch = case["n"], case["qbits"], case["batch"]
    if kind == "ntt":
        return {"a": _uniform(g, batch, n, modulus(bits))}
    if kind == "crypt":
        return {"m": torch.randint(0, case["t"], (batch, n), generator=g, device=DEV, dtype=torch.int64)}
    return pairs(n, bits, batch, kind == "he")


def _scheme(n, bits, t, key):
    """A scheme with installed keys, uniform as public and evaluation keys are."""
    y = cy.Yashe(n, modulus(bits), t)
    key = _host(key)
    y.set_keys(key[0], key[1], key[2:])
    return y


def prepare(case, seed):
    kind, x = case["kind"], _inputs(case, seed)
    if kind == "mixed":
        groups, jobs = [], []
        for (n, bits, t), d in zip(MIXED, x):
            y = _scheme(n, bits, t, d["key"])
            out = y.ring.empty(case["per_class"])
            groups.append(out)
            jobs.append([("yashe", y, d["a"][j:j + 1], d["b"][j:j + 1], out[j:j + 1], True)
                         for j in range(case["per_class"])])
        plan = MixedPlan([j for row in zip(*jobs) for j in row])  # the classes take turns
        return {"kind": kind, "plan": plan, "out": groups}
    n, q, batch = case["n"], modulus(case["qbits"]), case["batch"]
    if kind == "mul":
        ring = cy.Ring(n, q)
        return dict(x, kind=kind, ring=ring, out=ring.empty(batch))
    if kind == "he":
        y = _scheme(n, case["qbits"], case["t"], x.pop("key"))
        return dict(x, kind=kind, y=y, out=y.ring.empty(batch), relin=case["relin"])
    if kind == "ntt":
        ring = cy.Ring(n, q)
        return {"kind": kind, "ring": ring, "res": ring.crt(x["a"]), "inverse": case["inverse"]}
    if kind == "crypt":
        y = cy.Yashe(n, q, case["t"])
        y.keygen(int(seed) + 1)
        return dict(x, kind=kind, y=y, seed=int(seed) + 7, ct=y.ring.empty(batch))
    raise ValueError(kind)


def run(state):
    kind = state["kind"]
    if kind == "mul":
        return state["ring"].polymul(state["a"], state["b"], out=state["out"])
    if kind == "he":
        return state["y"].mul(state["a"], state["b"], relin=state["relin"], out=state["out"])
    if kind == "ntt":  # in place, as the entry point works
        return state["ring"].ntt(state["res"], inverse=state["inverse"])
    if kind == "crypt":
        ct = state["y"].encrypt(state["m"], state["seed"], out=state["ct"])
        return {"ct": ct, "m": state["y"].decrypt(ct)}
    state["plan"].launch()
    return state["out"]


# ---- what a pass cannot do without ---------------------------------------------------
def _primes(bits):
    return math.ceil(bits / 30)


def _transforms(case):
    """Length-N transforms of one pass, with as many 30-bit primes as the exact integers need."""
    n, bits = case["n"], case["qbits"]
    logn, ell = int(math.log2(n)), math.ceil(bits / 32)
    product = _primes(2 * bits + logn)
    kind = case["kind"]
    if kind == "ntt":
        return product * case["batch"]
    if kind == "mul":
        return 3 * product * case["batch"]
    if kind == "crypt":
        return 4 * product * case["batch"]  # the key's transforms are the same for all
    relin = (ell + 1) * _primes(bits + 32 + logn + math.log2(ell)) if case["relin"] else 0
    return (3 * product + relin) * case["batch"]


def work(case):
    """Bytes: operands read and results written once. Operations: the transforms' butterflies, a modular
    product (3 integer operations) and two sums each."""
    if case["kind"] == "mixed":
        parts = [work({"kind": "he", "n": n, "qbits": bits, "relin": True, "batch": case["per_class"]})
                 for n, bits, _ in MIXED]
        return {k: sum(p[k] for p in parts) for k in ("bytes", "flops")}
    n, bits, batch = case["n"], case["qbits"], case["batch"]
    poly = 8 * n * ((bits + 63) // 64)
    if case["kind"] == "ntt":
        moved = 2 * 4 * n * _transforms(case)
    elif case["kind"] == "crypt":
        moved = batch * (2 * poly + 2 * 8 * n)
    else:
        moved = 3 * poly * batch
        if case.get("relin"):
            moved += math.ceil(bits / 32) * poly
    return {"bytes": moved, "flops": 5 * _transforms(case) * n * int(math.log2(n)) // 2}


# ---- exact results in integers ---------------------------------------------------------
def _ints(x):
    """[n][limbs] words -> list of integers."""
    raw = _host(x).astype("<u8").tobytes()
    w = 8 * x.shape[-1]
    return [int.from_bytes(raw[i:i + w], "little") for i in range(0, len(raw), w)]


def _negacyclic(a, b):
    """a b modulo x^n + 1 over the integers, by one long product (signed coefficients)."""
    n = len(a)
    most = n * max(map(abs, a), default=0) * max(map(abs, b), default=0)
    w = (most.bit_length() + 2 + 7) // 8

    def pack(v):
        pos = b"".join((x if x > 0 else 0).to_bytes(w, "little") for x in v)
        neg = b"".join((-x if x < 0 else 0).to_bytes(w, "little") for x in v)
        return int.from_bytes(pos, "little") - int.from_bytes(neg, "little")

    half = 1 << (8 * w - 1)
    shift = int.from_bytes(half.to_bytes(w, "little") * (2 * n), "little")
    raw = (pack(a) * pack(b) + shift).to_bytes(2 * n * w + 1, "little")
    c = [int.from_bytes(raw[i * w:(i + 1) * w], "little") - half for i in range(2 * n)]
    return [c[i] - c[i + n] for i in range(n)]


def _limbs(polys, q):
    limbs = (q.bit_length() + 63) // 64
    raw = b"".join(x.to_bytes(8 * limbs, "little") for p in polys for x in p)
    return np.frombuffer(raw, dtype="<i8").reshape(len(polys), -1, limbs).copy()


def exact(case, seed):
    kind = case["kind"]
    if kind in ("mixed", "ntt"):
        return None  # too long in integers; the transform's order and roots are the library's own
    n, q = case["n"], modulus(case["qbits"])
    if kind == "crypt":
        return {"ct": None, "m": _inputs(case, seed)["m"].cpu()}  # decryption gives the plaintexts back
    products = 1 + (math.ceil(case["qbits"] / 32) if case.get("relin") else 0)
    if case["batch"] * products * (n * case["qbits"] / 5e5) ** 1.6 * 0.15 > 10:
        return None
    s = _inputs(case, seed)
    out = []
    for j in range(case["batch"]):
        a, b = _ints(s["a"][j]), _ints(s["b"][j])
        if kind == "he":
            h = (q - 1) // 2
            a, b = ([x - q if x > h else x for x in v] for v in (a, b))
            c = [((case["t"] * x + h) // q) % q for x in _negacyclic(a, b)]
            if case["relin"]:
                evk = [_ints(e) for e in s["key"][2:]]
                parts = [_negacyclic([(x >> (32 * d)) & 0xFFFFFFFF for x in c], e) for d, e in enumerate(evk)]
                c = [sum(col) % q for col in zip(*parts)]
        else:
            c = [x % q for x in _negacyclic(a, b)]
        out.append(c)
    return torch.from_numpy(_limbs(out, q))
