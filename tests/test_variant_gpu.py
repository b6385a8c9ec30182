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


# chunk sizes on either side of the lines at which a default chunk with the FP32 pre-pass changes its kernel
@pytest.mark.parametrize("n", [4095, 4096, 8191, 8192, (1 << 16) - 1, 1 << 16, 1 << 17, (1 << 19) - 1, 1 << 19])
@pytest.mark.parametrize("policy,depth", [(0, 0), (0, 1), (2, 2)])
@pytest.mark.parametrize("family", [0, 1, 3, 5])
def test_fp32_chunks_agree_whatever_their_kernel(cp, family, policy, depth, n):
    p, q = cp.Prover(), cp.Prover()
    q.set_level_variant(family, cp.FP32_PREFILTER, 1)  # one kernel for every size
    lo, hi, dp = p.random_boxes(family, n, seed=n, max_label=2)
    kw = dict(policy=policy, max_depth=depth, precision=cp.FP32_PREFILTER, digest=1, level_capacity=1 << 22)
    a, b = (x.refine_boxes(family, lo, hi, dp, engine=cp.ENGINE_LEVELS, **kw) for x in (p, q))
    for k in ("evaluated", "unresolved", "clipped", "fp32_decided", "handles_evaluated", "verdicts", "per_depth", "digest"):
        assert a[k] == b[k], k
    assert a["evaluated"] > 0
    p.close()
    q.close()


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("n,depth", [(31, 2), (4095, 1), (4095, 2), (4096, 1), (4096, 2), (20000, 5)])
@pytest.mark.parametrize("family", range(6))
def test_static_call_agrees_with_the_level_loop(cp, family, n, depth, precision):
    p = cp.Prover()
    lo, hi, dp = p.random_boxes(family, n, seed=n, max_label=4)
    a = cp.refine_boxes_static(family, lo, hi, dp, precision=precision, max_depth=depth)
    b = p.refine_boxes(family, lo, hi, dp, precision=precision, max_depth=depth, policy=cp.SPLIT_WIDEST)
    for k in ("evaluated", "unresolved", "clipped", "fp32_decided", "handles_evaluated", "verdicts", "per_depth"):
        assert a[k] == b[k], k
    p.close()


@pytest.mark.parametrize("n,depth", [(1 << 16, 1), ((1 << 16) + 1, 1), (1 << 14, 2), ((1 << 14) + 1, 2), (100, 0)])
@pytest.mark.parametrize("family", [0, 2])
def test_fp32_graph_agrees_whatever_its_shape(cp, family, n, depth):
    p = cp.Prover()
    lo, hi, dp = p.random_boxes(family, n, seed=n, max_label=2)
    kw = dict(max_depth=depth, policy=cp.SPLIT_UNIFORM, precision=cp.FP32_PREFILTER, digest=1, level_capacity=1 << 20,
              engine=cp.ENGINE_GRAPH)
    a, b = p.refine_boxes(family, lo, hi, dp, **kw), p.refine_boxes(family, lo, hi, dp, block=1024, **kw)
    for k in ("evaluated", "unresolved", "clipped", "fp32_decided", "handles_evaluated", "verdicts", "per_depth", "digest"):
        assert a[k] == b[k], k
    p.close()
