"""The FP64 filter where its error bound is tight: reciprocal seeds off by the 2^-19 that the bound
assumes, either way, and boxes on the boundary between proved and critical."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

from tests import boxgen
from tests.test_filter_cpu import FULL, HANDLES, HERE, MASK, ROOT, VERDICT, _boxes, _filter, decide_mask


@pytest.fixture(scope="module", params=["0x1p-19", "-0x1p-19"])
def filt(request, tmp_path_factory):
    so = str(tmp_path_factory.mktemp("filter") / "libfilter.so")
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-shared", "-fPIC",
                    f"-DCPF_SEED_ERROR={request.param}", "-I" + os.path.join(ROOT, "circlepacking_b200", "csrc"),
                    os.path.join(HERE, "filter_host.cpp"), "-o", so], check=True)
    return ctypes.CDLL(so)


def _boundary(oracle, family):
    """Boxes between a proved and a critical one of the same lattice, bisected to the last bit, and the
    same moved along the way by 2^-52 to 2^-24 of it."""
    lo, hi = _boxes(oracle, family, "step", 6000)
    v, _ = oracle.eval_boxes(family, lo, hi)
    a, b = np.flatnonzero(v == oracle.PROVED), np.flatnonzero(v == oracle.CRITICAL)
    if not a.size or not b.size:
        return lo, hi
    rng = np.random.default_rng(40 + family)
    a, b = rng.choice(a, 1500), rng.choice(b, 1500)
    at = lambda t: (lo[:, a] + t * (lo[:, b] - lo[:, a]), hi[:, a] + t * (hi[:, b] - hi[:, a]))
    t0, t1 = np.zeros(1500), np.ones(1500)  # proved at t0, not proved at t1
    for _ in range(54):
        t = 0.5 * (t0 + t1)
        proved = oracle.eval_boxes(family, *at(t))[0] == oracle.PROVED
        t0, t1 = np.where(proved, t, t0), np.where(proved, t1, t)
    off = [0.0] + [s * 2.0 ** -k for k in range(52, 23, -4) for s in (-1, 1)]
    out = [at(t + o) for t in (t0, t1) for o in off]
    return np.concatenate([x[0] for x in out], 1), np.concatenate([x[1] for x in out], 1)


@pytest.mark.parametrize("kind", ["boundary", "coarse", "reference", "thin", "sub"])
@pytest.mark.parametrize("family", range(6))
def test_bound_holds_with_the_worst_seeds(oracle, filt, family, kind):
    lo, hi = _boundary(oracle, family) if kind == "boundary" else _boxes(oracle, family, kind)
    verdict, mask = oracle.eval_boxes(family, lo, hi)
    crit = (mask & 0x3F).astype(np.uint8)
    if kind == "boundary":
        assert (verdict == oracle.PROVED).any() and (verdict == oracle.CRITICAL).any()
    for need in (VERDICT, HANDLES, MASK, FULL):
        for order in (0, 1) if need in (HANDLES, MASK) else (0,):
            decided, got = _filter(filt, family, need, lo, hi, order)
            trap = decided & ((mask & 0x80) != 0)  # (in DECIDE order a failing first handle may stand ahead of it)
            assert not trap.any() or (need != FULL and family > 2 and (got[trap] != 0).all())
            decided &= ~trap
            if need <= HANDLES:
                assert ((got != 0) == (crit != 0))[decided].all()
            else:
                assert (got == (crit if need == FULL else decide_mask(family, crit, order)))[decided].all()
