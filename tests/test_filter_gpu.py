"""The FP64 filter on the device: its seeds over every operand, and the filtered
evaluation against the unfiltered one (a trace request turns the filter off)."""
import numpy as np
import pytest
import torch

from tests import boxgen
from tests.test_filter_cpu import _boxes, decide_mask

pytestmark = pytest.mark.gpu


def test_seed_errors(cp):
    """Both approximations stay within 2^-19, the error bound's assumption."""
    out = torch.zeros(2, dtype=torch.float64, device="cuda")
    assert cp.lib().cp_seed_error(cp._ptr(out), cp._stream()) == 0
    assert (out.cpu().numpy() < 2.0 ** -19).all(), out


@pytest.mark.parametrize("kind", ["coarse", "step", "reference", "narrow", "thin", "sub", "points", "wild"])
@pytest.mark.parametrize("family", range(6))
def test_filtered_evaluation_matches_directed(cp, oracle, family, kind):
    lo, hi = _boxes(oracle, family, kind, 60000)
    v0, m0, tr = (x.cpu().numpy() for x in cp.eval_boxes(family, lo, hi, trace=True))
    v, m = (x.cpu().numpy() for x in cp.eval_boxes(family, lo, hi))
    assert (v == v0).all() and (m == m0).all()
    clean = (m0 & 0x80) == 0  # DECIDE may stop ahead of a trap site
    for order in (0, 1):
        o = np.full(lo.shape[1], order, np.uint8)
        v, m = (x.cpu().numpy() for x in cp.eval_boxes(family, lo, hi, mode=cp.EVAL_DECIDE, order=o))
        assert (v == v0)[clean].all()
        want = decide_mask(family, (m0 & 0x3F).astype(np.uint8), order) | (m0 & 0x40)
        if family > 2:
            want = np.where(v0 == cp.NOFIT, np.uint8(0x40), want)
        assert (m == want)[clean].all()


@pytest.mark.parametrize("family", range(6))
def test_handles_match_directed(cp, oracle, family):
    """handles_evaluated of a refinement that ends at its seeds, against the
    criteria a trace shows as evaluated up to the first failing one."""
    lo, hi = _boxes(oracle, family, "reference", 60000)
    v0, m0, tr = (x.cpu().numpy() for x in cp.eval_boxes(family, lo, hi, trace=True))
    keep = (v0 <= 1)
    lo, hi, m0, tr = lo[:, keep], hi[:, keep], m0[keep], tr[keep]
    if family == 0:
        done = ~np.isnan(tr[:, :2, 0])
        n = done[:, 0].astype(int) + (done[:, 1] & ~(done[:, 0] & ((m0 & 1) != 0)))
    elif family in (1, 2):
        n = np.ones(lo.shape[1], int)
    else:
        n = np.where((m0 & (3 if family == 3 else 1)) != 0, 1, 2)
    p = cp.Prover()
    try:
        for engine in (cp.ENGINE_LEVELS, cp.ENGINE_GRAPH):
            r = p.refine_boxes(family, lo, hi, max_depth=0, engine=engine, level_capacity=1 << 16)
            assert r["evaluated"] == lo.shape[1]
            assert r["handles_evaluated"] == n.sum()
    finally:
        p.close()
