"""Choices of schedules: number 0 is the default, which depends on a call's size; what the autotuner measures
holds for calls of the measured regime, what an import names without one for all."""
import pytest

from oracle import ring

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


def test_choice_of_a_regime(cy):
    """At N = 16384 the default is schedule 3 (block pairs) for small calls."""
    _choose(cy, 0)
    default = {b: cy.tuning_schedule(16384, 6, "mul", b) for b in BLOCKS}
    assert default[1] == 3 and default[2000] != 3
    cy.tuning_import("n16384.l6.mul=2@3")
    assert {b: cy.tuning_schedule(16384, 6, "mul", b) for b in BLOCKS} == {
        b: 2 if v == 3 else v for b, v in default.items()}
    cy.tuning_import("n16384.l6.mul=4@%d;n16384.l6.mul=0@3" % default[2000])
    assert {b: cy.tuning_schedule(16384, 6, "mul", b) for b in BLOCKS} == {
        b: 3 if v == 3 else 4 for b, v in default.items()}
    spec = cy.tuning_export()
    cy.tuning_import("n16384.l6.mul=1")  # no regime: every size, and the choices for regimes are gone
    assert {cy.tuning_schedule(16384, 6, "mul", b) for b in BLOCKS} == {1}
    assert "n16384.l6.mul=1;" in cy.tuning_export() and "n16384.l6.mul=4@" not in cy.tuning_export()
    cy.tuning_import(spec)
    assert cy.tuning_schedule(16384, 6, "mul", 1) == 3 and cy.tuning_schedule(16384, 6, "mul", 2000) == 4
    for bad in ("n16384.l6.mul=1@-1", "n16384.l6.mul=1@99"):
        with pytest.raises(cy.CyError):
            cy.tuning_import(bad)


def test_tuning_a_batch_leaves_single_calls_alone(cy):
    _choose(cy, 0)
    n, q = 16384, ring.largest_prime_below(2**62, 2**16)
    default = {op: cy.tuning_schedule(n, 1, op, 5) for op in ("mul", "mulc", "ks")}
    y = cy.Yashe(n, q, 17)
    y.autotune(batch=64)
    assert {op: cy.tuning_schedule(n, 1, op, 5) for op in default} == default
    for op in default:
        assert ("n16384.l1.%s=" % op) in cy.tuning_export()


def test_the_autotuner_times_each_kernel_once(cy):
    """N = 8192 has three product kernels and two transforms under numbers 0 .. 3: a check and three timed
    runs of each, two launches per run."""
    r = cy.Ring(8192, ring.largest_prime_below(2**62, 2**16))
    before = cy.launch_count()
    r.autotune(batch=1)
    assert cy.launch_count() - before == 4 * 2 * (3 + 2)


def test_refused(cy):
    for n, l, op, b in ((1000, 1, "mul", 1), (1024, 0, "mul", 1), (1024, 7, "mul", 1), (1024, 1, "add", 1),
                        (1024, 1, "mul", -1), (32768, 1, "mul", 1)):
        with pytest.raises(cy.CyError):
            cy.tuning_schedule(n, l, op, b)
