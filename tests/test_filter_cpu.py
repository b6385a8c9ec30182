"""The FP64 filter (csrc/cp_filter.cuh), built for the host, against the CPU
restatement of the directed evaluation: every box it decides has the same
failing criteria and reaches no trap site, for lattice boxes from coarse to
very narrow, random sub-boxes, degenerate and out-of-domain boxes."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

from tests import boxgen

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)
VERDICT, HANDLES, MASK, FULL = range(4)


@pytest.fixture(scope="module")
def filt(tmp_path_factory):
    so = str(tmp_path_factory.mktemp("filter") / "libfilter.so")
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-shared", "-fPIC",
                    "-I" + os.path.join(ROOT, "circlepacking_b200", "csrc"), os.path.join(HERE, "filter_host.cpp"),
                    "-o", so], check=True)
    return ctypes.CDLL(so)


def _filter(filt, family, need, lo, hi, order=0):
    lo, hi = np.ascontiguousarray(lo), np.ascontiguousarray(hi)
    n = lo.shape[1]
    decided, mask = np.zeros(n, np.uint8), np.zeros(n, np.uint8)
    filt.filter_boxes(family, need, lo.ctypes.data_as(ctypes.c_void_p), hi.ctypes.data_as(ctypes.c_void_p),
                      ctypes.c_long(n), order, decided.ctypes.data_as(ctypes.c_void_p),
                      mask.ctypes.data_as(ctypes.c_void_p))
    return decided.astype(bool), mask


def decide_mask(family, full, order):
    """The mask DECIDE order reports: the first failing sub-criterion in its order."""
    bits = {3: (2, 3, 0, 1) if order else (0, 1, 2, 3), 4: (1, 0) if order else (0, 1),
            5: (1, 0) if order else (0, 1)}.get(family, (0, 1))
    out = np.zeros_like(full)
    for b in reversed(bits):
        out = np.where(full & (1 << b), np.uint8(1 << b), out)
    return out


def _boxes(oracle, family, kind, n=20000):
    d = boxgen.DIMS[family]
    sizes = {"coarse": (8, 8, 8, 8), "step": (64, 64, 64, 64), "reference": (256, 256, 256, 64),
             "narrow": (1000, 30, 30, 1), "thin": (100000, 30, 20, 1)}.get(kind, (64, 32, 32, 16))[:d]
    idx = np.random.default_rng(family).integers(0, int(np.prod(sizes)), n)
    lo, hi = oracle.lattice_boxes(family, boxgen.LAMBDA, sizes, idx)
    if kind == "sub":
        lo, hi = boxgen.sub_boxes(lo, hi, 31 + family)
    if kind == "points":
        lo, hi = boxgen.point_boxes(lo, hi, 32 + family)
    if kind == "wild":  # out of the domain, overlapping and disordered radii, special values
        rng = np.random.default_rng(33 + family)
        s = rng.uniform(-0.2, 0.3, lo.shape) * (rng.random(lo.shape) < 0.3)
        lo, hi = lo + s, hi + s + rng.uniform(0, 0.3, lo.shape) * (rng.random(lo.shape) < 0.2)
        for bad in (np.nan, np.inf, -np.inf, 0.0, 1.0, 5e-324, 1e300):
            lo[rng.integers(0, d, 50), rng.integers(0, n, 50)] = bad
            hi[rng.integers(0, d, 50), rng.integers(0, n, 50)] = bad
    return lo, hi


@pytest.mark.parametrize("kind", ["coarse", "step", "reference", "narrow", "thin", "sub", "points", "wild"])
@pytest.mark.parametrize("family", range(6))
def test_filter_decides_as_the_directed_evaluation(oracle, filt, family, kind):
    lo, hi = _boxes(oracle, family, kind)
    verdict, mask = oracle.eval_boxes(family, lo, hi)
    crit = (mask & 0x3F).astype(np.uint8)
    for need in (VERDICT, HANDLES, MASK, FULL):
        for order in (0, 1) if need in (HANDLES, MASK) else (0,):
            decided, got = _filter(filt, family, need, lo, hi, order)
            # no box at a trap site; in DECIDE order a failing first handle returns ahead of the second one's
            trap = decided & ((mask & 0x80) != 0)
            assert not trap.any() or (need != FULL and family > 2 and (got[trap] != 0).all())
            decided &= ~trap
            assert not (decided & (verdict == oracle.EMPTY)).any()
            if need <= HANDLES:
                assert ((got != 0) == (crit != 0))[decided].all()
            else:
                want = crit if need == FULL else decide_mask(family, crit, order)
                assert (got == want)[decided].all()
    if kind in ("step", "reference"):  # the filter does its work on the ordinary boxes
        assert decided[verdict <= 1].mean() > 0.99


def test_filter_asin(filt):
    rng = np.random.default_rng(1)
    d = np.exp(rng.uniform(-8, 1, 200000))
    x = np.concatenate([rng.uniform(-1, 1, 100000), 1 - 2.0 ** -rng.uniform(1, 15.9, 50000),
                        2.0 ** -rng.uniform(0, 40, 50000)])
    n = x * d
    out, ok = np.zeros_like(n), np.zeros(n.size, np.uint8)
    p = lambda a: a.ctypes.data_as(ctypes.c_void_p)
    filt.filter_asin(p(n), p(d), ctypes.c_long(n.size), p(out), p(ok))
    q = n.astype(np.longdouble) / d
    want = np.arcsin(q)
    # polynomial 9.8e-13, seeds 2^-24 here: the square is below 2^-46; 1 - |q| as exact as n and d
    assert ok[np.abs(q) < 1 - 2.0 ** -15.9].all()
    assert np.abs(out - want).max() < 3e-12
