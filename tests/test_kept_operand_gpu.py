"""Encryption and decryption run their products with the keys' kept transforms (two jobs per
block): odd and even batches, one (the ordinary product), every number of limbs, new keys in the
same scheme; values at the edges of [0, q). Decryption against exact integers, encryption against
one ciphertext at a time."""
import random

import pytest

from oracle import ring

pytestmark = pytest.mark.gpu


def _decrypt(f, c, q, t):
    x = ring.polymul_mod(f, c, q)
    return [((t * v + (q - 1) // 2) // q) % t for v in x]


@pytest.mark.parametrize("bits", [62, 127, 190, 250, 310, 380])
@pytest.mark.parametrize("n", [512, 1024, 2048])
def test_decrypt_batches(bits, n):
    import torch

    import cuyashe_gb300 as cy

    rng = random.Random(bits + n)
    q, t = (1 << bits) - 57, 1024
    q -= 1 - q % 2
    y = cy.Yashe(n, q, t)

    def poly():
        return [rng.choice([0, 1, q - 1, rng.randrange(q)]) for _ in range(n)]

    for _ in range(2):  # the second keys replace the first
        f = poly()
        y.set_keys([f], [poly()], [poly() for _ in range(y.ell)])
        for batch in (1, 2, 3):
            c = [poly() for _ in range(batch)]
            m = y.decrypt(y.ring.upload(c)).cpu()
            torch.cuda.synchronize()
            for j in range(batch):
                assert m[j].tolist() == _decrypt(f, c[j], q, t)


@pytest.mark.parametrize("n,bits", [(1024, 190), (4096, 127), (8192, 62), (16384, 380)])
def test_encrypt_with_kept_key_equals_product(n, bits):
    """A batch's ciphertexts equal h s + e + Delta m with h s computed by the ordinary product:
    zero plaintexts, and the same draws with a scheme whose h is 0 give e alone."""
    import torch

    import cuyashe_gb300 as cy

    rng = random.Random(n)
    q, t, batch = (1 << bits) - 57, 17, 3
    y, z, w = cy.Yashe(n, q, t), cy.Yashe(n, q, t), cy.Yashe(n, q, t)
    h = [rng.randrange(q) for _ in range(n)]
    one = [1] + [0] * (n - 1)
    evk = [[0] * n for _ in range(y.ell)]
    y.set_keys([one], [h], evk)
    z.set_keys([one], [[0] * n], evk)  # h = 0: e
    w.set_keys([one], [one], evk)      # h = 1: s + e
    m = torch.zeros((batch, n), dtype=torch.int64, device="cuda")
    ct, e, se = (s.encrypt(m, 5) for s in (y, z, w))
    s = y.ring.polysub(se, e)
    hh = y.ring.upload([h] * batch)
    assert torch.equal(ct, y.ring.polyadd(y.ring.polymul(hh, s), e))


@pytest.mark.parametrize("n,bits", [(1024, 62), (2048, 310), (4096, 127), (8192, 250), (16384, 190)])
def test_encrypt_one_equals_first_of_batch(n, bits):
    """Draws are counted per ciphertext, so a batch begins with the ciphertext of a call of one; h at
    the edges of [0, q)."""
    import torch

    import cuyashe_gb300 as cy

    rng = random.Random(n)
    q = (1 << bits) - 57
    y = cy.Yashe(n, q, 17)
    h = [rng.choice([0, 1, q - 1]) for _ in range(n)]
    y.set_keys([[1] + [0] * (n - 1)], [h], [[0] * n for _ in range(y.ell)])
    m = torch.randint(17, (5, n), generator=torch.Generator().manual_seed(n)).cuda()
    whole = y.encrypt(m, seed=11)
    for batch in (1, 2, 4):
        assert torch.equal(y.encrypt(m[:batch].contiguous(), seed=11), whole[:batch])
