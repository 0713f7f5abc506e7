"""Tensor products and keyswitches of four- and five-limb moduli (an even and an odd number of 32-bit
words each) in the kernels of their own, N >= 1024, under every schedule: coefficients next to (q - 1)/2
and of full and empty words, keys of q - 1. Exact: the results must equal the oracle's."""
import random

import pytest

from oracle.yashe import Yashe as OYashe, YasheKeys, YasheParams

pytestmark = pytest.mark.gpu


def _edge_poly(n, q, rng):
    words = (q.bit_length() + 31) // 32
    h = (q - 1) // 2
    out = []
    for _ in range(n):
        x = sum(rng.choice([0, 2**32 - 1, rng.randrange(2**32)]) << (32 * i) for i in range(words))
        out.append(rng.choice([0, 1, q - 1, q - 2, h - 1, h, h + 1, x % q, x % q]))
    return out


def _numbers(cy, n, limbs, op):
    for v in range(64):
        try:
            cy.tuning_import("n%d.l%d.%s=%d" % (n, limbs, op, v))
        except cy.CyError:
            return
        yield v


@pytest.mark.parametrize("bits", [224, 250, 288, 320])
@pytest.mark.parametrize("n", [1024, 2048])
def test_tensor_and_keyswitch(bits, n):
    import torch

    import cuyashe_gb300 as cy

    rng = random.Random(bits + n)
    q, t = (1 << bits) - rng.choice([1, 3, 5]), 1024
    y = cy.Yashe(n, q, t)
    L = y.ring.L
    o = OYashe(YasheParams(n=n, q=q, t=t, w_bits=32))
    assert y.ell == o.p.ell == (bits + 31) // 32
    a, b = _edge_poly(n, q, rng), _edge_poly(n, q, rng)
    evk = [[q - 1 if (i + d) % 3 else rng.randrange(q) for i in range(n)] for d in range(y.ell)]
    keys = YasheKeys(f=[1] + [0] * (n - 1), h=[0] * n, evk=evk)
    y.set_keys([keys.f], [keys.h], evk)
    A, B = y.ring.upload([a, b, a]), y.ring.upload([b, b, b])
    tensor = [o.mul_tensor(a, b), o.mul_tensor(b, b)]
    switched = [o.keyswitch(keys, a), o.keyswitch(keys, b)]
    relin = [o.keyswitch(keys, c) for c in tensor]
    try:
        for v in _numbers(cy, n, L, "mulc"):
            got = y.ring.download(y.mul(A, B, relin=False))
            torch.cuda.synchronize()
            assert [list(x) for x in got] == [tensor[0], tensor[1], tensor[0]], "tensor, schedule %d" % v
        for v in _numbers(cy, n, L, "ks"):
            got = y.ring.download(y.keyswitch(A))
            assert [list(x) for x in got] == [switched[0], switched[1], switched[0]], "keyswitch, schedule %d" % v
            got = y.ring.download(y.mul(A, B))  # its digits limb-major
            torch.cuda.synchronize()
            assert [list(x) for x in got] == [relin[0], relin[1], relin[0]], "multiply, schedule %d" % v
    finally:
        cy.tuning_import("n%d.l%d.mulc=0;n%d.l%d.ks=0" % (n, L, n, L))
