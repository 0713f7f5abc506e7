"""The schedule a mixed plan starts with: one block per SM for a short list, two for a long one,
with the same products either way."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("jobs,schedule", [(3, 1), (4000, 0)])
def test_schedule_by_length(jobs, schedule):
    import cuyashe_gb300 as cy

    n, q = 1024, (1 << 62) - 57
    R = cy.Ring(n, q)
    g = torch.Generator(device="cuda")
    g.manual_seed(jobs)
    a, b = (torch.randint(0, q, (jobs, n, 1), generator=g, device="cuda", dtype=torch.int64) for _ in range(2))
    out = R.empty(jobs)
    plan = cy.MixedPlan([("mul", R, a[j:j + 1], b[j:j + 1], out[j:j + 1]) for j in range(jobs)])
    assert plan.schedule == schedule
    ref = R.polymul(a, b)
    for s in (schedule, 1 - schedule):
        plan.schedule = s
        out.zero_()
        plan.launch()
        plan.status()
        assert torch.equal(out, ref)
