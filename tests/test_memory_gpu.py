"""A graph-engine refinement on a device that is nearly full."""
import pytest
import torch

from tests.test_refine_gpu import _same

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("left", [48 << 20, 160 << 20])
def test_fewer_warps_where_memory_is_short(cp, left):
    """The stacks of all warps at this depth and shape take 580 MB; with less left the refinement runs on
    fewer warps, with the same report."""
    lo = torch.tensor([[0.6], [0.12], [0.08], [0.05]], dtype=torch.float64, device="cuda")
    hi = lo + torch.tensor([[0.05], [0.06], [0.06], [0.05]], dtype=torch.float64, device="cuda")
    depth = torch.full((1,), 52, dtype=torch.uint8, device="cuda")  # split ten times
    args = 3, lo, hi, depth
    kw = dict(policy=cp.SPLIT_WIDEST, max_depth=62, digest=1, level_capacity=1 << 16, block=1024)
    p = cp.Prover()
    want = p.refine_boxes(*args, engine=cp.ENGINE_LEVELS, **kw)
    _same(p.refine_boxes(*args, engine=cp.ENGINE_GRAPH, **kw), want)
    p.close()
    p = cp.Prover()
    torch.cuda.empty_cache()
    fill = torch.empty(torch.cuda.mem_get_info()[0] - left, dtype=torch.uint8, device="cuda")
    try:
        got = p.refine_boxes(*args, engine=cp.ENGINE_GRAPH, **kw)
    finally:
        del fill
        torch.cuda.empty_cache()
        p.close()
    _same(got, want)
    assert want["evaluated"] > 64
