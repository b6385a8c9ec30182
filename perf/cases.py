"""Workloads of the lane-packing prover, through its public Python entry points.

A case is a dict of plain values.  `listed()` names the ones that stand for the
real uses, `draw(rng)` gives more of the same ranges, `prepare(case, seed)` builds
what a program holds before the call, `run(state)` is one pass, and `work(case)`
the bytes and operations that pass cannot do without.

Kinds (the key "kind"):
  eval       per-box verdicts of boxes in device memory (cp_eval_boxes)
  lattice    refinement of a lattice seed (cp_refine)
  boxes      refinement of explicit seed boxes in device or host memory
             (cp_refine_boxes, cp_refine_boxes_host)
  static     refinement in the library's fixed scratch (cp_refine_boxes_static)
  proof      full-domain proof of a family, or one rank's share of it (cp_prove_family)
  reference  the reference's lambda queue over lattice launches (cp_prove_family_reference)
  gradient   one forward and backward pass of the proposal network (cp_model_loss_grad_kind)
"""
from __future__ import annotations

import numpy as np
import torch

import circlepacking_b200 as cp

# Operations per box on the reference kernel's early-exit path (adds, multiplies,
# divisions and arcsines counted as one each), rounded from the CPU restatement's
# counts on lattice seeds refined uniformly.
OPS_PER_BOX = (275, 125, 295, 360, 162, 395)
# Boxes evaluated per seed box when a 64^dims lattice over the whole domain is
# bisected on every axis once and twice (measured).
GROWTH = ((1.0, 12.7, 141.0), (1.0, 7.3, 43.0), (1.0, 12.6, 128.0), (1.0, 12.0, 119.0), (1.0, 7.2, 41.0),
          (0.6, 2.6, 17.0))
# Boxes a whole proof evaluates with the library's settings, per family.
PROOF_BOXES = (489e6, 8.4e6, 130e6, 3.64e6, 10.5e6, 0.278e6)

# Inputs and outputs of the proposal network's layers.
LAYERS = ((16, 64), (64, 64), (64, 8))


def listed():
    return [
        # a handful of boxes checked interactively or by another program: launch latency
        dict(name="eval_small", kind="eval", family=cp.START_END_2D, n=1000, full=True, precision=cp.FP64),
        # verdicts and complete masks of a large ragged box set
        dict(name="eval_full_middle", kind="eval", family=cp.MIDDLE, n=1_000_003, full=True, precision=cp.FP64),
        # the benchmark's step for one family: 64^4 lattice, two uniform levels, graph engine
        dict(name="lattice_middle", kind="lattice", family=cp.MIDDLE, size=64, depth=2, engine=cp.ENGINE_GRAPH,
             precision=cp.FP64, digest=False),
        # the default engine (host-driven levels), with the verdict digest that proofs are compared by
        dict(name="lattice_start_levels", kind="lattice", family=cp.START, size=33, depth=2, engine=cp.ENGINE_LEVELS,
             precision=cp.FP64, digest=True),
        # the FP32 pre-pass option
        dict(name="lattice_fp32", kind="lattice", family=cp.START_END_3D, size=31, depth=2, engine=cp.ENGINE_GRAPH,
             precision=cp.FP32_PREFILTER, digest=False),
        # seed boxes handed over in host memory: the whole call with its copies
        dict(name="boxes_host", kind="boxes", family=cp.END_3D, n=1_500_001, depth=2, policy=cp.SPLIT_UNIFORM,
             engine=cp.ENGINE_LEVELS, host=True),
        # boxes of uneven depth and size in one device worklist, binary splits
        dict(name="boxes_uneven", kind="boxes", family=cp.START_END_3D, n=3_000_017, depth=5, policy=cp.SPLIT_WIDEST,
             engine=cp.ENGINE_GRAPH, host=False),
        # the call for programs that let no library allocate: small, many levels
        dict(name="static_small", kind="static", family=cp.END_2D, n=4096, depth=6, precision=cp.FP64),
        # the largest proof, one graph launch per lambda slab
        dict(name="proof_start", kind="proof", family=cp.START, engine=cp.ENGINE_GRAPH, parts=2),
        # the smallest proof, one host round trip per level
        dict(name="proof_end_3d_levels", kind="proof", family=cp.END_3D, engine=cp.ENGINE_LEVELS, parts=2),
        # the reference's own loop, many lattice launches
        dict(name="reference_middle", kind="reference", family=cp.MIDDLE, size=48, launches=48),
        # a batch of labelled boxes through the proposal network and back
        dict(name="gradient_middle", kind="gradient", family=cp.MIDDLE, n=65536),
    ]


def _log_int(rng, lo, hi):
    return int(round(lo * (hi / lo) ** rng.random()))


def draw(rng):
    kind = rng.choice(("eval", "eval", "lattice", "lattice", "lattice", "boxes", "boxes", "static", "proof", "reference",
                       "gradient"))
    family = rng.randrange(6)
    engine = rng.choice((cp.ENGINE_LEVELS, cp.ENGINE_GRAPH))
    precision = rng.choice((cp.FP64, cp.FP64, cp.FP32_PREFILTER))
    if kind == "eval":
        return dict(kind=kind, family=family, n=_log_int(rng, 200, 4_000_000), full=rng.random() < 0.5,
                    precision=precision)
    if kind == "lattice":
        wide = cp.DIMS[family] == 4
        return dict(kind=kind, family=family, size=_log_int(rng, 8, 44) if wide else _log_int(rng, 12, 160),
                    depth=rng.randrange(3), engine=engine, precision=precision, digest=rng.random() < 0.5)
    if kind == "boxes":
        policy = rng.choice((cp.SPLIT_UNIFORM, cp.SPLIT_LAMBDA, cp.SPLIT_WIDEST, cp.SPLIT_HYBRID))
        return dict(kind=kind, family=family, n=_log_int(rng, 1000, 3_000_000),
                    depth=rng.randint(1, 2) if policy == cp.SPLIT_UNIFORM else rng.randint(2, 6), policy=policy,
                    engine=engine, host=rng.random() < 0.4)
    if kind == "static":
        return dict(kind=kind, family=family, n=_log_int(rng, 50, 20_000), depth=rng.randint(1, 6), precision=precision)
    if kind == "proof":
        return dict(kind=kind, family=family, engine=engine, parts=rng.choice((2, 3, 4, 5, 8, 13)))
    if kind == "reference":
        return dict(kind=kind, family=family, size=_log_int(rng, 24, 64), launches=rng.randint(8, 64))
    return dict(kind=kind, family=family, n=_log_int(rng, 64, 131072))


def _jitter(seed, lo=cp.LAMBDA_MIN, hi=cp.LAMBDA_MAX):
    """A lambda range inside [lo, hi], its ends moved in by up to 2% of it."""
    r = np.random.RandomState(seed % (1 << 31))
    a, b = r.random_sample(2) * 0.02 * (hi - lo)
    return float(lo + a), float(hi - b)


def _rows(case, seed):
    """Parameters of a fresh network and labelled feature rows (9 features, 7 zero columns)."""
    family, n = case["family"], case["n"]
    r = np.random.RandomState(seed % (1 << 31))
    params = []
    for k, (i, o) in enumerate(LAYERS):
        w = r.uniform(-1, 1, (i, o)) / np.sqrt(9 if k == 0 else i)
        if k == 0:
            w[9:] = 0
        params += [w.reshape(-1), r.uniform(-1, 1, o) / np.sqrt(9 if k == 0 else i)]
    feats = np.zeros((n, 16), np.float32)
    feats[:, :9] = r.uniform(-1, 1, (n, 9))
    crit = r.randint(0, 1 << cp.N_CRITERIA[family], n).astype(np.uint8)
    axis = r.randint(-1, cp.DIMS[family], n).astype(np.int8)
    return np.concatenate(params).astype(np.float32), feats, crit, axis


class _State:
    pass


def prepare(case, seed):
    s = _State()
    s.case, s.seed = case, seed
    kind, family = case["kind"], case["family"]
    dims = cp.DIMS[family]
    if kind not in ("eval", "gradient"):
        s.prover = cp.Prover()
    if kind == "eval":
        # boxes of the reference's lattice, at random places
        sizes = cp.REFERENCE_SIZES[family]
        total = int(np.prod([int(x) for x in sizes], dtype=np.int64))
        g = torch.Generator(device="cuda").manual_seed(seed)
        index = torch.randint(0, total, (case["n"],), generator=g, device="cuda", dtype=torch.int64)
        s.lo, s.hi = cp.lattice_boxes(family, _jitter(seed), sizes, index)
    elif kind == "lattice":
        s.opts = dict(seed_sizes=[case["size"]] * dims, seed_lambda=_jitter(seed), max_depth=case["depth"],
                      precision=case["precision"], engine=case["engine"], digest=case["digest"],
                      level_capacity=0 if case["size"] ** dims > 1 << 23 else 1 << 24)
    elif kind in ("boxes", "static"):
        s.lo, s.hi, s.depth = s.prover.random_boxes(family, case["n"], seed=seed, max_label=min(8, case["depth"] + 2))
        if kind == "boxes":
            if case["host"]:
                s.lo, s.hi, s.depth = (x.cpu().numpy() for x in (s.lo, s.hi, s.depth))
            s.opts = dict(max_depth=case["depth"], policy=case["policy"], engine=case["engine"], level_capacity=1 << 24)
    elif kind == "proof":
        s.opts = dict(engine=case["engine"], digest=1, seed_parts=case["parts"], seed_part=seed % case["parts"])
    elif kind == "reference":
        lo, hi = _jitter(seed, 0.5, 0.75)
        s.opts = dict(la_lb=lo, la_ub=hi, sizes=[2 * case["size"]] + [case["size"]] * (dims - 1),
                      max_launches=case["launches"], trace_cap=case["launches"])
    elif kind == "gradient":
        s.rows = _rows(case, seed)
    return s


def _report(r, digest=False):
    """What a refinement found; its launches and times are no results."""
    keys = [k for k in ("evaluated", "unresolved", "clipped", "fp32_decided", "handles_evaluated", "max_depth_seen",
                        "proved", "slabs_done", "first_unresolved_slab") if k in r]
    out = dict(counts=np.array([int(r[k]) for k in keys], np.int64), verdicts=np.array(r["verdicts"], np.int64),
               per_depth=np.array((list(r["per_depth"]) + [0] * 64)[:64], np.int64))
    if digest:
        out["digest"] = np.array([[d & 0xFFFFFFFF, d >> 32] for d in r["digest"]], np.int64)
    return out


def run(s):
    c = s.case
    kind, family = c["kind"], c["family"]
    if kind == "eval":
        return cp.eval_boxes(family, s.lo, s.hi, precision=c["precision"],
                             mode=cp.EVAL_FULL if c["full"] else cp.EVAL_DECIDE)
    if kind == "lattice":
        return _report(s.prover.refine(family, **s.opts), c["digest"])
    if kind == "boxes":
        return _report(s.prover.refine_boxes(family, s.lo, s.hi, s.depth, **s.opts))
    if kind == "static":
        return _report(cp.refine_boxes_static(family, s.lo, s.hi, s.depth, precision=c["precision"],
                                              max_depth=c["depth"]))
    if kind == "proof":
        return _report(s.prover.prove_family(family, **s.opts), True)
    if kind == "reference":
        r = s.prover.prove_family_reference(family, **s.opts)
        # (boxes_evaluated depends on how far past the failing slab the blocks had run)
        return dict(trace=np.array(r["trace"]), remaining=np.array(r["remaining"]),
                    counts=np.array([int(r["proved"]), r["launches"]], np.int64))
    loss, grad = cp.model_loss_grad(family, *s.rows, kind=1)
    return dict(loss=loss, grad=grad)


def work(case):
    kind, family = case["kind"], case["family"]
    dims, ops = cp.DIMS[family], OPS_PER_BOX[family]
    box = 16 * dims
    if kind == "eval":
        return {"bytes": case["n"] * (box + 2), "flops": case["n"] * ops}
    if kind == "lattice":
        seeds = case["size"] ** dims
        return {"bytes": 1024, "flops": int(seeds * GROWTH[family][case["depth"]] * ops)}
    if kind in ("boxes", "static"):
        # with random labels about half of the boxes are above the depth limit
        grown = case["n"] * (1 + 0.5 * case["depth"])
        return {"bytes": case["n"] * (box + 1), "flops": int(grown * ops)}
    if kind == "proof":
        return {"bytes": 1024, "flops": int(PROOF_BOXES[family] / case["parts"] * ops)}
    if kind == "reference":
        # a launch stops at the first failing lambda slab, most often among its first few
        return {"bytes": 1024, "flops": int(case["launches"] * 2 * case["size"] ** (dims - 1) * ops)}
    # forward, data and weight gradients
    weights = sum(a * b for a, b in LAYERS)
    return {"bytes": case["n"] * (16 * 4 + 2) + 8 * cp.model_param_count(), "flops": case["n"] * 2 * 3 * weights}


def exact(case, seed):
    """Loss and gradient of the proposal network in 64 bits.  Every other result is
    a whole number (verdicts, masks, counts, digests), or the reference loop's
    lambda bounds, which follow from directed rounding."""
    if case["kind"] != "gradient":
        return None
    family, n = case["family"], case["n"]
    params, feats, crit, axis = _rows(case, seed)
    w, b, at = [], [], 0
    for i, o in LAYERS:
        w.append(params[at:at + i * o].reshape(i, o).astype(np.float64))
        b.append(params[at + i * o:at + i * o + o].astype(np.float64))
        at += i * o + o
    x, h = [feats.astype(np.float64)], []
    for k in range(3):
        h.append(x[k] @ w[k] + b[k])
        u = np.tanh(np.sqrt(2 / np.pi) * (h[k] + 0.044715 * h[k] ** 3))
        x.append(0.5 * h[k] * (1 + u))
    z, crits, dims = h[2], min(cp.N_CRITERIA[family], 4), cp.DIMS[family]
    y = ((crit[:, None] >> np.arange(crits)) & 1).astype(np.float64)
    zc, za = z[:, :crits], z[:, 4:4 + dims]
    dz = np.zeros_like(z)
    dz[:, :crits] = (1 / (1 + np.exp(-zc)) - y) / n
    p = np.exp(za - za.max(axis=1, keepdims=True))
    p /= p.sum(axis=1, keepdims=True)
    rows = np.flatnonzero(axis >= 0)
    loss = ((np.logaddexp(0, zc) - y * zc).sum() - np.log(p[rows, axis[rows]]).sum()) / n
    p[rows, axis[rows]] -= 1
    dz[rows, 4:4 + dims] = p[rows] / n
    grads = []
    for k in (2, 1, 0):
        grads = [(x[k].T @ dz).reshape(-1), dz.sum(axis=0)] + grads
        if k:
            u = np.tanh(np.sqrt(2 / np.pi) * (h[k - 1] + 0.044715 * h[k - 1] ** 3))
            slope = 0.5 * (1 + u) + 0.5 * h[k - 1] * (1 - u * u) * np.sqrt(2 / np.pi) * (1 + 3 * 0.044715 * h[k - 1] ** 2)
            dz = dz @ w[k].T * slope
    return dict(loss=float(loss), grad=np.concatenate(grads))
