"""Choices of schedules: number 0 is the default, which depends on a call's size."""
import pytest

pytestmark = pytest.mark.gpu

LENGTHS = (1024, 2048, 4096, 8192, 16384)
BLOCKS = (1, 14, 70, 76, 77, 152, 153, 304, 305, 607, 608, 2000)


@pytest.fixture()
def cy():
    import cuyashe_gb300

    cuyashe_gb300.lib()
    yield cuyashe_gb300
    _choose(cuyashe_gb300, 0)


def _choose(cy, v, limbs=range(1, 7), ops=("mul", "mulc", "ks", "ntt")):
    cy.tuning_import(";".join("n%d.l%d.%s=%d" % (n, l, op, v) for n in LENGTHS for l in limbs for op in ops))


def _all(cy):
    return {(n, l, op, b): cy.tuning_schedule(n, l, op, b) for n in LENGTHS for l in range(1, 7)
            for op in ("mul", "mulc", "ks", "ntt") for b in BLOCKS}


def test_number_0_gives_the_default_back(cy):
    _choose(cy, 0)
    default = _all(cy)
    assert len({v for (n, _, op, _), v in default.items() if (n, op) == (16384, "mul")}) > 1  # it depends on the size
    _choose(cy, 1)
    assert set(_all(cy).values()) == {1}
    _choose(cy, 0)
    assert _all(cy) == default


def test_every_default_can_be_chosen_by_number(cy):
    _choose(cy, 0)
    for (n, l, op, b), v in _all(cy).items():
        assert v > 0
        cy.tuning_import("n%d.l%d.%s=%d" % (n, l, op, v))
        assert cy.tuning_schedule(n, l, op, 1) == cy.tuning_schedule(n, l, op, 10**6) == v
        cy.tuning_import("n%d.l%d.%s=0" % (n, l, op))


def test_refused(cy):
    for n, l, op, b in ((1000, 1, "mul", 1), (1024, 0, "mul", 1), (1024, 7, "mul", 1), (1024, 1, "add", 1),
                        (1024, 1, "mul", -1), (32768, 1, "mul", 1)):
        with pytest.raises(cy.CyError):
            cy.tuning_schedule(n, l, op, b)
