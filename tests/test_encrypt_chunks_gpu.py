"""Encryption over several launches: small words at the start of each output row, multiplied in the keyswitch
basis in place, pairs of ciphertexts per block, odd batches. Against the ordinary product of h and the
same s, and the first ciphertexts against a call of one launch."""
import random

import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,bits,batch", [(16384, 380, 61), (8192, 190, 201), (4096, 127, 601), (1024, 62, 2501)])
def test_chunked_encryption(n, bits, batch):
    import torch

    import cuyashe_gb300 as cy

    rng = random.Random(n)
    q, t = (1 << bits) - 57, 17
    y, z, w = cy.Yashe(n, q, t), cy.Yashe(n, q, t), cy.Yashe(n, q, t)
    h = [rng.choice([0, q - 1, rng.randrange(q)]) for _ in range(n)]
    one = [1] + [0] * (n - 1)
    evk = [[0] * n for _ in range(y.ell)]
    y.set_keys([one], [h], evk)
    z.set_keys([one], [[0] * n], evk)  # h = 0: e + Delta m
    w.set_keys([one], [one], evk)      # h = 1: s + e + Delta m
    m = torch.randint(t, (batch, n), generator=torch.Generator().manual_seed(n)).cuda()
    with cy.Trace() as tr:
        ct = y.encrypt(m, 5)
    assert sum(v[0] for k, v in tr.kernels.items() if k.startswith("mul_key")) > 1  # several launches
    e, se = z.encrypt(m, 5), w.encrypt(m, 5)
    s = y.ring.polysub(se, e)
    H = y.ring.upload([h])
    for j in range(0, batch, 100):
        part = s[j:j + 100].contiguous()
        expected = y.ring.polyadd(y.ring.polymul(H.expand(part.shape[0], -1, -1).contiguous(), part),
                                  e[j:j + 100].contiguous())
        assert torch.equal(ct[j:j + 100], expected)
    assert torch.equal(y.encrypt(m[:5].contiguous(), 5), ct[:5])
