"""The schedules that calls run by default, at the sizes on both sides of each line of the rule: batches of a few
polynomials repeated, against the oracle."""
import random

import pytest

from oracle import ring
from oracle.yashe import Yashe as OYashe, YasheKeys, YasheParams

pytestmark = pytest.mark.gpu


def _lines(cy, n, limbs, op, k, most):
    """Batches next to each change of the default schedule, and one."""
    number = [cy.tuning_schedule(n, limbs, op, j * k) for j in range(1, most + 1)]
    jobs = {1}
    for j in range(1, most):
        if number[j] != number[j - 1]:
            jobs |= {j, j + 1}
    return sorted(jobs)


# (operations whose oracle takes seconds at N = 16384 are left to the smaller modulus)
@pytest.mark.parametrize("n,bits,ops", [(1024, 62, "mul mulc ks"), (2048, 127, "mul mulc ks"), (4096, 127, "mul mulc ks"),
                                        (8192, 62, "mul mulc ks"), (16384, 62, "mul mulc ks"), (16384, 300, "mul")])
def test_both_sides_of_each_line(n, bits, ops):
    import torch

    import cuyashe_gb300 as cy

    rng = random.Random(n + bits)
    q, t = ring.largest_prime_below(2**bits, 2**16), 17
    o = OYashe(YasheParams(n=n, q=q, t=t, w_bits=32))
    y = cy.Yashe(n, q, t)
    R = y.ring

    def poly():
        return [rng.randrange(q) for _ in range(n)]

    keys = YasheKeys(f=poly(), h=poly(), evk=[poly() for _ in range(y.ell)])
    y.set_keys([keys.f], [keys.h], keys.evk)
    pa, pb = [poly(), poly()], [poly(), poly()]
    A, B = R.upload(pa), R.upload(pb)
    info = y.info()
    calls = {
        "mul": (R.k, lambda a, b: R.polymul(a, b), lambda i: ring.polymul_mod(pa[i], pb[i], q)),
        "mulc": (info.tensor_primes, lambda a, b: y.mul(a, b, relin=False), lambda i: o.mul_tensor(pa[i], pb[i])),
        "ks": (info.relin_primes, lambda a, b: y.keyswitch(a), lambda i: o.keyswitch(keys, pa[i])),
    }
    cy.tuning_import(";".join("n%d.l%d.%s=0" % (n, R.L, op) for op in ("mul", "mulc", "ks")))
    for op in ops.split():
        k, call, exact = calls[op]
        expected = R.upload([exact(0), exact(1)])
        for jobs in _lines(cy, n, R.L, op, k, 160):
            pick = torch.tensor([rng.randrange(2) for _ in range(jobs)], device="cuda")
            out = call(A[pick].contiguous(), B[pick].contiguous())
            assert torch.equal(out, expected[pick]), (op, jobs)


@pytest.mark.parametrize("n", [1024, 2048, 4096, 8192, 16384])
def test_transforms(n):
    """The standalone transform under its default against schedule 1, and back."""
    import torch

    import cuyashe_gb300 as cy

    R = cy.Ring(n, ring.largest_prime_below(2**62, 2**16))
    cy.tuning_import("n%d.l1.ntt=0" % n)
    primes = torch.tensor([int(p) for p in R.primes], dtype=torch.int64).view(1, -1, 1)
    for jobs in _lines(cy, n, 1, "ntt", R.k, 200):
        g = torch.Generator().manual_seed(jobs)
        x = (torch.randint(0, 2**40, (jobs, R.k, n), generator=g) % primes).to(torch.int32).cuda()
        here, other = x.clone(), x.clone()
        R.ntt(here)
        cy.tuning_import("n%d.l1.ntt=1" % n)
        R.ntt(other)
        cy.tuning_import("n%d.l1.ntt=0" % n)
        assert torch.equal(here, other)
        R.ntt(here, inverse=True)
        assert torch.equal(here, x)
