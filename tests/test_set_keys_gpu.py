"""Installing keys: every kept form of them is made in few launches, and replaced by later keys (also for
calls recorded or prepared before)."""
import random

import pytest

from oracle.yashe import Yashe as OYashe, YasheKeys, YasheParams

pytestmark = pytest.mark.gpu


def _keys(rng, n, q, ell):
    def poly():
        return [rng.randrange(q) for _ in range(n)]

    return YasheKeys(f=poly(), h=poly(), evk=[poly() for _ in range(ell)])


@pytest.mark.parametrize("n,bits", [(512, 127), (1024, 62), (4096, 127), (8192, 190)])
def test_launches(n, bits):
    """f^2 (product and epilogue), then split, transform and scaling of f and f^2 together and of h and the
    evaluation key together (h's split apart), and the key's second layout at N = 4096."""
    import cuyashe_gb300 as cy

    rng = random.Random(n)
    q = (1 << bits) - 57
    y = cy.Yashe(n, q, 17)
    k = _keys(rng, n, q, y.ell)
    for _ in range(2):
        before = cy.launch_count()
        y.set_keys([k.f], [k.h], k.evk)
        assert cy.launch_count() - before <= 10


def test_recorded_and_prepared_multiplies_follow_new_keys():
    import torch

    import cuyashe_gb300 as cy

    n, q, t = 1024, (1 << 127) - 57, 1024
    rng = random.Random(3)
    o = OYashe(YasheParams(n=n, q=q, t=t, w_bits=32))
    y = cy.Yashe(n, q, t)
    a, b = ([rng.randrange(q) for _ in range(n)] for _ in range(2))
    A, B = y.ring.upload([a]), y.ring.upload([b])
    out, out2 = y.ring.empty(1), y.ring.empty(1)
    graph = plan = None
    for _ in range(2):
        k = _keys(rng, n, q, y.ell)
        y.set_keys([k.f], [k.h], k.evk)
        if graph is None:
            graph, plan = y.mul_graph(A, B, out), cy.MixedPlan([("yashe", y, A, B, out2, True)])
        graph.launch()
        plan.launch()
        torch.cuda.synchronize()
        expected = o.mul(k, a, b, relin=True)
        assert list(y.ring.download(out)[0]) == expected
        assert list(y.ring.download(out2)[0]) == expected
