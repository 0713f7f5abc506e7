"""Calls of several launches (residue scratch of about 24 MiB each): batches that divide evenly,
unevenly and with one job over, against the same jobs in calls of a single launch. All
operations, bit for bit."""
import random

import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,bits,batches", [(16384, 380, (11, 20, 21, 41)), (8192, 190, (61, 121)), (4096, 127, (513,))])
def test_chunked_calls_equal_single_launches(n, bits, batches):
    import torch

    import cuyashe_gb300 as cy

    rng = random.Random(n + bits)
    q = (1 << bits) - 57
    y = cy.Yashe(n, q, 17)

    def poly():
        return [rng.randrange(q) for _ in range(n)]

    y.set_keys([poly()], [poly()], [poly() for _ in range(y.ell)])
    pool = y.ring.upload([poly() for _ in range(4)])
    gen = torch.Generator().manual_seed(n)
    for batch in batches:
        a = pool[torch.randint(4, (batch,), generator=gen).cuda()].contiguous()
        b = pool[torch.randint(4, (batch,), generator=gen).cuda()].contiguous()
        calls = {
            "product": lambda i, j: y.ring.polymul(a[i:j], b[i:j]),
            "tensor": lambda i, j: y.mul(a[i:j], b[i:j], relin=False),
            "multiply": lambda i, j: y.mul(a[i:j], b[i:j]),
            "keyswitch": lambda i, j: y.keyswitch(a[i:j]),
            "decrypt": lambda i, j: y.decrypt(a[i:j]),
        }
        for name, call in calls.items():
            whole = call(0, batch)
            parts = torch.cat([call(i, min(i + 5, batch)) for i in range(0, batch, 5)])
            assert torch.equal(whole, parts), (name, batch)
