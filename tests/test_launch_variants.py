"""Selection of the launch variants (no kernel runs): the launch-size rule of 2 to 5 species,
a caller's choice over it, and a variant read and set back."""
import pytest

from particleclem_b200 import abi, autotune, hydro, native

FORMS = [abi.PREC_FP64, abi.PREC_FP64_FAST, abi.PREC_MIXED]
STAGES = autotune.TUNED_STAGES + (autotune.TAIL_STAGE,)
SIZES = (0, 1, 592, 593, 1184, 1185, 1 << 30)
FLUX2 = 5


def _table(prec, ns):
    lib = native.load()
    return {(st, n): lib.pcg_launch_variant_for(prec, ns, st, n) for st in range(7) for n in SIZES}


@pytest.mark.parametrize("ns", [1, 2, 3, 9, 21])
@pytest.mark.parametrize("prec", FORMS)
def test_a_variant_read_and_set_back_changes_nothing(prec, ns):
    if ns not in hydro.species_counts():
        pytest.skip(f"library built without {ns} species")
    before = _table(prec, ns)
    for st in STAGES:
        autotune.set_variant(prec, ns, st, autotune.get_variant(prec, ns, st))
    assert _table(prec, ns) == before
    saved = {st: autotune.get_variant(prec, ns, st) for st in STAGES}
    for st in STAGES:
        for v in range(autotune.n_variants(prec, st)):
            autotune.set_variant(prec, ns, st, v)
            assert autotune.get_variant(prec, ns, st) == v
            if v != saved[st]:  # a caller's choice holds at every size
                assert {native.load().pcg_launch_variant_for(prec, ns, st, n) for n in SIZES} == {v}
        autotune.set_variant(prec, ns, st, saved[st])
    assert _table(prec, ns) == before


def test_few_species_take_other_caps_up_to_the_rules_size():
    if 3 not in hydro.species_counts():
        pytest.skip("library built without 3 species")
    t = _table(abi.PREC_FP64, 3)
    assert t[FLUX2, 1184] == 0 and t[FLUX2, 1185] == 2
    t = _table(abi.PREC_MIXED, 3)
    assert t[FLUX2, 592] == 1 and t[FLUX2, 593] == 2


def test_bad_queries_are_refused():
    lib = native.load()
    for bad in ((-1, 3, 0, 1), (3, 3, 0, 1), (0, 64, 0, 1), (0, 9, 7, 1), (0, 9, -1, 1), (0, 9, 0, -1)):
        assert lib.pcg_launch_variant_for(*bad) == -1
