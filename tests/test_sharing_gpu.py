"""The depth-first kernel's work sharing where hardly any refinement takes it: waits that run out
(further launches over what was left), parcel slots used again, stacks that spill, launch
numbers that come back.  Every refinement against the level by level loop, box by box."""
import pytest
import torch

from tests.test_refine_gpu import _same

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def prover(cp):
    p = cp.Prover()
    yield p
    p.close()


def _one_box(cp, prover):
    """One box split 14 times: every parent but the first warp's is shared work."""
    lo = torch.tensor([[0.6], [0.12], [0.08], [0.05]], dtype=torch.float64, device="cuda")
    hi = lo + torch.tensor([[0.05], [0.06], [0.06], [0.05]], dtype=torch.float64, device="cuda")
    return (3, lo, hi, None), dict(max_depth=14, policy=cp.SPLIT_WIDEST)


def _many(cp, prover):
    """Seeds of uneven depth for every warp."""
    lo, hi, dp = prover.random_boxes(2, 40000, seed=5, max_label=3)
    return (2, lo, hi, dp), dict(max_depth=10, policy=cp.SPLIT_WIDEST)


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("polls,slots,strict", [(0, -1, -1), (1, 3, 32), (-1, 1, 32), (-1, 64, 0), (-1, -1, 64)])
@pytest.mark.parametrize("seeds", [_one_box, _many])
def test_limits_do_not_change_the_refinement(cp, prover, seeds, polls, slots, strict, precision):
    args, kw = seeds(cp, prover)
    kw.update(precision=precision, digest=1, level_capacity=1 << 22)
    prover.set_deep_limits(polls, slots, strict)
    try:
        a = prover.refine_boxes(*args, engine=cp.ENGINE_GRAPH, **kw)
        s = prover.deep_stats()
    finally:
        prover.set_deep_limits()
    _same(a, prover.refine_boxes(*args, engine=cp.ENGINE_LEVELS, **kw))
    assert a["launches"] == s["launches"]
    if polls in (0, 1) and seeds is _one_box:
        assert s["launches"] > 1, s  # nobody waited: what was given away took further launches
    if 0 < slots < 64 and seeds is _one_box:
        assert s["parcels"] > slots, s
    if seeds is _many:
        assert s["spilled"] > 0, s


def test_launch_numbers_start_over(cp, prover):
    args, kw = _one_box(cp, prover)
    kw.update(digest=1, level_capacity=1 << 20)
    want = prover.refine_boxes(*args, engine=cp.ENGINE_LEVELS, **kw)
    epochs = []
    prover.set_deep_limits(slots=2, epoch=(1 << 23) - 7)
    for _ in range(4):
        _same(prover.refine_boxes(*args, engine=cp.ENGINE_GRAPH, **kw), want)
        epochs.append(prover.deep_stats()["epoch"])
    prover.set_deep_limits()
    assert epochs[0] >= (1 << 23) - 4 and 2 <= epochs[-1] < 1 << 20, epochs


@pytest.mark.parametrize("limits", [(1 << 20, -1, -1), (-1, 0, -1), (-1, 4097, -1), (-1, -1, 4097)])
def test_limits_out_of_range_are_refused(cp, prover, limits):
    with pytest.raises(cp.ProverError, match="CP_ERR_INVALID"):
        prover.set_deep_limits(*limits)
