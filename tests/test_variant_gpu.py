"""Which variant of the level kernel a chunk runs: a choice of the caller or of the autotuner
holds for chunks of every size; only the default looks at the size."""
import pytest

pytestmark = pytest.mark.gpu

SIZES = (1, (1 << 16) - 1, 1 << 16, 1 << 24)


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("family", range(6))
def test_chosen_variant_holds_for_every_chunk(cp, family, precision):
    p = cp.Prover()
    default = [p.get_level_variant(family, precision, n) for n in SIZES]
    assert default[0] == default[1] == 1 and default[2] == default[3] > 1
    for v in range(4):
        p.set_level_variant(family, precision, v)
        assert [p.get_level_variant(family, precision, n) for n in SIZES] == [v] * 4
    other = 1 - precision
    assert p.get_level_variant(family, other, 1) == 1  # the other precision keeps its default
    p.close()


def test_autotuned_variant_holds_for_every_chunk(cp):
    p = cp.Prover()
    best, ms = p.autotune(cp.END_2D, seed_sizes=[8, 8, 8], max_depth=1)
    assert [p.get_level_variant(cp.END_2D, 0, n) for n in SIZES] == [best] * 4
    p.close()
