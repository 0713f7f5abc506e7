"""CRT split of the product kernels: coefficients at the edges of their words.

Products, and HE multiplies (centred operands), of polynomials whose coefficients are
0, 1, q - 1, the two values next to (q - 1)/2, and values whose 32-bit words are all
zeros or all ones, at every number of limbs: the sums of the split then reach the ends
of their ranges. Exact integers: the results must equal the oracle's.
"""
import random

import pytest

from oracle import ring
from oracle.yashe import Yashe as OYashe, YasheParams

pytestmark = pytest.mark.gpu


def _edge_poly(n, q, rng):
    words = (q.bit_length() + 31) // 32
    h = (q - 1) // 2
    out = []
    for _ in range(n):
        x = sum(rng.choice([0, 2**32 - 1, rng.randrange(2**32)]) << (32 * i) for i in range(words))
        out.append(rng.choice([0, 1, q - 1, q - 2, h, h + 1, x % q, x % q]))
    return out


@pytest.mark.parametrize("bits", [30, 33, 64, 96, 127, 128, 190, 192, 250, 256, 320, 380, 384])
@pytest.mark.parametrize("n", [8, 1024])
def test_products_of_edge_coefficients(bits, n):
    import torch

    import cuyashe_gb300 as cy

    rng = random.Random(bits * 7 + n)
    q = (1 << bits) - rng.choice([1, 3, 5])  # all words of q - 1 full but the lowest
    R = cy.Ring(n, q)
    a, b = _edge_poly(n, q, rng), _edge_poly(n, q, rng)
    out = R.download(R.polymul(R.upload([a]), R.upload([b])))
    torch.cuda.synchronize()
    assert list(out[0]) == ring.polymul_mod(a, b, q)
    if n > 8:
        return
    t = 17
    oy = OYashe(YasheParams(n=n, q=q, t=t, w_bits=32))
    y = cy.Yashe(n, q, t)
    out = y.ring.download(y.mul(y.ring.upload([a]), y.ring.upload([b]), relin=False))
    torch.cuda.synchronize()
    assert list(out[0]) == oy.mul_tensor(a, b)


@pytest.mark.parametrize("bits", [62, 127, 250, 380])
def test_residues_of_edge_coefficients(bits):
    import torch

    import cuyashe_gb300 as cy

    rng = random.Random(bits)
    n, q = 64, (1 << bits) - 1
    R = cy.Ring(n, q)
    a = _edge_poly(n, q, rng)
    res = R.crt(R.upload([a])).cpu().numpy()
    torch.cuda.synchronize()
    for i, p in enumerate(R.primes):
        assert [int(v) for v in res[0, i]] == [x % p for x in a]


@pytest.mark.parametrize("bits", [31, 62, 95, 127, 160, 190, 224, 250, 288, 320, 352, 380])
def test_largest_products(bits):
    """All coefficients q - 1: the product's coefficients run from -(n - 2)(q - 1)^2 to
    n (q - 1)^2, the ends of the range the ICRT's estimate of the multiple of M must
    resolve; every number of 32-bit words of q."""
    import torch

    import cuyashe_gb300 as cy

    n, q = 256, (1 << bits) - 1
    R = cy.Ring(n, q)
    a = [q - 1] * n
    out = R.download(R.polymul(R.upload([a]), R.upload([a])))
    torch.cuda.synchronize()
    assert list(out[0]) == ring.polymul_mod(a, a, q)
