"""The depth-first kernel (graph engine) against the level by level loop at the edges of
its buffers, and the FP32 pre-pass's decisions against pinned ones."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

COUNTS = ("evaluated", "unresolved", "clipped", "fp32_decided", "handles_evaluated", "verdicts", "per_depth", "digest")


def _same(a, b):
    for k in COUNTS:
        assert list(np.atleast_1d(a[k])) == list(np.atleast_1d(b[k])), k


# seeds: one, around a warp, around a parcel and the first pieces of all warps
@pytest.mark.parametrize("n", [1, 31, 33, 2369, 4097])
@pytest.mark.parametrize("policy,depth", [(0, 2), (2, 9)])
@pytest.mark.parametrize("precision", [0, 1])
def test_depth_first_matches_levels(cp, n, policy, depth, precision):
    p = cp.Prover()
    lo, hi, dp = p.random_boxes(2, n, seed=n + 1, max_label=3)
    if n > 31:
        dp[::7] = 255  # dropped seeds
    kw = dict(max_depth=depth, policy=policy, precision=precision, digest=1, level_capacity=1 << 20)
    _same(p.refine_boxes(2, lo, hi, dp, engine=cp.ENGINE_GRAPH, **kw),
          p.refine_boxes(2, lo, hi, dp, engine=cp.ENGINE_LEVELS, **kw))


@pytest.mark.parametrize("block", [64, 128, 256, 512, 1024])
def test_depth_first_spills(cp, block):
    """One box split 14 times: stacks far beyond the part on chip, and parcels."""
    lo = torch.tensor([[0.6], [0.12], [0.08], [0.05]], dtype=torch.float64, device="cuda")
    hi = lo + torch.tensor([[0.05], [0.06], [0.06], [0.05]], dtype=torch.float64, device="cuda")
    prover = cp.Prover()
    kw = dict(max_depth=14, policy=cp.SPLIT_WIDEST, digest=1, level_capacity=1 << 20)
    a = prover.refine_boxes(3, lo, hi, None, engine=cp.ENGINE_GRAPH, block=block, **kw)
    b = prover.refine_boxes(3, lo, hi, None, engine=cp.ENGINE_LEVELS, **kw)
    assert a["evaluated"] > 64
    _same(a, b)


# evaluated, FP32-decided and guarded criteria of a 7^4 (24^3) lattice and two uniform
# levels, from the shadow's general collision chain alone
PINNED = [(165429, 161812, 3617), (636378, 635717, 661), (167792, 164446, 3346), (165429, 165426, 3),
          (639189, 638721, 802), (82669, 82169, 617)]


@pytest.mark.parametrize("family", range(6))
def test_fp32_decisions_pinned(cp, family):
    sizes = [7] * 4 if cp.DIMS[family] == 4 else [24] * 3
    r = cp.Prover().refine(family, seed_sizes=sizes, max_depth=2, precision=cp.FP32_PREFILTER, engine=cp.ENGINE_LEVELS)
    assert (r["evaluated"], r["fp32_decided"], r["handles_evaluated"]) == PINNED[family]
