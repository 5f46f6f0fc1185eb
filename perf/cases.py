"""The work a user of this framework has it do, as timed cases.

Each case is one call sequence through the package's public entry points, on
seeded synthetic sequences of the shapes the package's own workloads and tests
use (``parflexdtw_b200.workloads``): 12-d chroma-like or 128-d Gaussian
frames, the second sequence a warped, noisy copy of the first.

``kind`` names the entry points:

* ``features``: one pair from device features, ``tiled_stage1_from_features``
  then ``run_stage2_from_tiled``;
* ``cost``: the drop-in ``parflex(C)`` on a cost matrix, on the device or as
  the NumPy array the reference's callers hold;
* ``batch``: many uneven pairs through a kept ``Batch`` (load, run, results,
  paths), in FP64 or in the FP32 form;
* ``pruned``: many long pairs through a kept ``PrunedBatch`` (learned tile
  pruning);
* ``untiled``: ``flexdtw`` on a whole cost matrix (D, P, B to the host);
* ``train``: one training step of the tile proposer (pooled map, forward,
  backward, Adam).
"""
import math
import random

import numpy as np
import torch

import parflexdtw_b200 as pfx
from parflexdtw_b200 import workloads
from parflexdtw_b200.prune import POOL, STRIDES, TileProposer

STEPS = ((1, 1), (1, 2), (2, 1))
WEIGHTS = (2.0, 3.0, 3.0)
BETA = 0.1
POS_WEIGHT, LR = 8.0, 2e-3


def listed():
    return [
        # the smallest calls: a 400 x 610 pair cut into many small tiles
        {"name": "cost_397x610_L100", "kind": "cost", "n": 397, "m": 610, "L": 100,
         "host": False},
        # one short recording against another, from features
        {"name": "features_2000x2400_L500", "kind": "features", "n": 2000, "m": 2400, "L": 500},
        # the drop-in call on a NumPy cost matrix: the upload is part of it
        {"name": "cost_host_2600x3101_L1000", "kind": "cost", "n": 2600, "m": 3101, "L": 1000,
         "host": True},
        # a pair of ordinary length at the reference's default tile length
        {"name": "cost_12000x13501_L4000", "kind": "cost", "n": 12000, "m": 13501, "L": 4000,
         "host": False},
        # one long pair, fewer tiles than the GPU has SMs
        {"name": "features_30000x37001_L4000", "kind": "features", "n": 30000, "m": 37001,
         "L": 4000},
        # one long pair, several tiles per SM
        {"name": "features_36000x41003_L2000", "kind": "features", "n": 36000, "m": 41003,
         "L": 2000},
        # a collection of uneven pairs, FP64
        {"name": "batch24_fp64", "kind": "batch", "pairs": 24, "lo": 2000, "hi": 20000, "d": 12,
         "L": 2000, "precision": "fp64"},
        # many short 128-d pairs, the FP32 form with the tensor-core cost
        {"name": "batch64_fp32_d128", "kind": "batch", "pairs": 64, "lo": 1000, "hi": 8000,
         "d": 128, "L": 1000, "precision": "fp32"},
        # a collection of long pairs with learned tile pruning
        {"name": "pruned6", "kind": "pruned", "pairs": 6, "lo": 24000, "hi": 36000, "L": 2000},
        # the accuracy baseline: the whole matrix as one tile, all of D, P, B
        {"name": "untiled_1500x1801", "kind": "untiled", "n": 1500, "m": 1801},
        # one step of training the tile proposer
        {"name": "train_20000x23001", "kind": "train", "n": 20000, "m": 23001, "L": 2000},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["cost", "cost", "features", "features", "features", "batch", "batch",
                       "pruned", "untiled", "train"])
    if kind == "cost":
        host = rng.random() < 0.3
        n = _log(rng, 397, 3000 if host else 12000)
        m = int(n * rng.uniform(0.7, 1.5))
        # 2 to 7 tiles per side, up to the reference's default tile length
        L = min(4000, max(40, int(min(n, m) / rng.uniform(1.5, 6.5))))
        return {"kind": kind, "n": n, "m": m, "L": L, "host": host}
    if kind == "features":
        n = _log(rng, 2000, 30000)
        m = int(n * rng.uniform(0.7, 1.25))
        return {"kind": kind, "n": n, "m": m,
                "L": rng.choice([x for x in (500, 1000, 1999, 2000, 4000) if x * 10 >= n])}
    if kind == "batch":
        if rng.random() < 0.5:
            return {"kind": kind, "pairs": rng.randint(3, 20), "lo": 2000,
                    "hi": _log(rng, 4000, 20000), "d": rng.choice([12, 12, 16, 24]),
                    "L": rng.choice([1000, 2000]), "precision": "fp64"}
        return {"kind": kind, "pairs": rng.randint(6, 60), "lo": 1000,
                "hi": _log(rng, 2000, 8000), "d": rng.choice([64, 100, 128]),
                "L": rng.choice([500, 1000]), "precision": "fp32"}
    if kind == "pruned":
        lo = rng.randint(15000, 24000)
        return {"kind": kind, "pairs": rng.randint(2, 5), "lo": lo,
                "hi": lo + rng.randint(1000, 10000), "L": 2000}
    if kind == "untiled":
        n = _log(rng, 300, 1500)
        return {"kind": kind, "n": n, "m": int(n * rng.uniform(0.7, 1.2))}
    n = _log(rng, 5000, 20000)
    return {"kind": kind, "n": n, "m": int(n * rng.uniform(0.7, 1.15)), "L": 2000}


def _shapes(case):
    """The lengths of a collection's pairs: the case's own, whatever the seed."""
    r = random.Random("%d %d %d" % (case["pairs"], case["lo"], case["hi"]))
    if case.get("precision") == "fp32":
        return [(r.randint(case["lo"], case["hi"]), r.randint(case["lo"], case["hi"]))
                for _ in range(case["pairs"])]
    return [(n, int(n * r.uniform(0.7, 1.4)))
            for n in (r.randint(case["lo"], case["hi"]) for _ in range(case["pairs"]))]


def _pair(rng, n, m, d=12):
    """(F1, F2) host features, d x n and d x m: chroma-like, or Gaussian latents."""
    F1, F2 = workloads.warped_pair(rng, n, m, d=d, noise=0.05 if d < 64 else 0.1,
                                   latent="dirichlet" if d < 64 else "gaussian")
    return F1, F2


def _features(case, seed):
    return _pair(np.random.default_rng(seed), case["n"], case["m"])


def _cost(case, seed):
    F1, F2 = (torch.from_numpy(f).cuda() for f in _features(case, seed))
    return 1.0 - F1.T @ F2


def _labels(case):
    """Tiles along the diagonal, as the tiles a path crosses."""
    hop = case["L"] - 1
    n1, n2 = -(-(case["n"] - 1) // hop), -(-(case["m"] - 1) // hop)
    lab = np.zeros((n1, n2), np.uint8)
    t = np.linspace(0, 1, 4 * (n1 + n2), endpoint=False)
    lab[(t * n1).astype(int), (t * n2).astype(int)] = 1
    return lab


def _padded(state, wp):
    """A path of K points as rows of the state's own fixed buffer: -1 past K."""
    out, k = state["wp"], wp.shape[0]
    out[:k] = wp
    out[k:] = -1
    return out


_geometry = None


def prepare(case, seed):
    global _geometry
    if case != _geometry:  # another shape: its pooled workspace, not the last one's
        pfx.clear_plan_cache()
        _geometry = dict(case)
    state = _prepare(case, seed)
    shapes = _shapes(case) if "pairs" in case else [(case["n"], case["m"])]
    # where run() puts the paths, which differ in length from input to input
    state["wp"] = np.empty((sum(n + m for n, m in shapes), 2), np.int64)
    return state


def _prepare(case, seed):
    kind = case["kind"]
    if kind == "features":
        return {"case": case, "F": [torch.from_numpy(f).cuda() for f in _features(case, seed)]}
    if kind in ("cost", "untiled"):
        C = _cost(case, seed)
        return {"case": case, "C": C.cpu().numpy() if case.get("host") else C}
    if kind == "train":
        net = TileProposer(seed=seed)
        net.init_optimizer()
        return {"case": case, "net": net, "label": _labels(case),
                "F": [torch.from_numpy(f).cuda() for f in _features(case, seed)]}
    rng = np.random.default_rng(seed)
    shapes = _shapes(case)
    d = case.get("d", 12)
    F = [tuple(torch.from_numpy(f).cuda() for f in _pair(rng, n, m, d)) for n, m in shapes]
    if kind == "batch":
        return {"case": case, "F": F,
                "batch": pfx.Batch(shapes, case["L"], STEPS, WEIGHTS, d,
                                   precision=case["precision"])}
    # room for the largest pair's cost: what a full-tile fallback needs
    room = max(int(1.2 * 8 * n * m) + (1 << 28) for n, m in shapes)
    return {"case": case, "F": F,
            "batch": pfx.PrunedBatch(shapes, case["L"], STEPS, WEIGHTS, d, cost_fma=True,
                                     wave_bytes=room)}


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "features":
        _, tiled = pfx.tiled_stage1_from_features(*state["F"], steps=STEPS, weights=WEIGHTS,
                                                  beta=BETA, L=case["L"])
        res = pfx.run_stage2_from_tiled(tiled, beta=BETA)
        return {"best": res["best_cost"], "end": res["best_end"],
                "wp": _padded(state, res["stitched_wp"])}
    if kind == "cost":
        best, wp = pfx.parflex(state["C"], STEPS, WEIGHTS, BETA, L=case["L"], profile_dir=None)
        return {"best": best, "wp": _padded(state, wp.T)}
    if kind == "batch":
        b = state["batch"]
        b.load(state["F"])
        b.run(BETA)
        best, end, lens = b.results()
        return {"best": best, "end": end, "len": lens,
                "wp": _padded(state, np.concatenate(b.paths(lens)))}
    if kind == "pruned":
        b = state["batch"]
        b.load(state["F"])
        out, info = b.run(BETA)
        return {"best": [x[0] for x in out], "len": [x[1].shape[1] for x in out],
                "wp": _padded(state, np.concatenate([x[1] for x in out], axis=1).T),
                "run": info["tiles_run"]}
    if kind == "untiled":
        best, wp, D, P, B, _ = pfx.flexdtw(state["C"], STEPS, WEIGHTS)
        return {"best": best, "wp": _padded(state, wp.T), "D": D, "P": P, "B": B}
    net = state["net"]
    pooled = net.pooled_cost(*state["F"])
    loss, grads = net.gradients(pooled, state["label"], case["n"], case["m"], case["L"],
                                POS_WEIGHT)
    net.step(grads, lr=LR)
    return {"loss": loss, "grads": grads, "params": net.params}


def work(case):
    """Bytes: the features or the cost matrix in, the path out.  Floating-point
    operations of a cell: 2 d + 1 for its cost, and for each of the three steps a
    product, two sums and a division (the kept tiles' share of them for a pruned
    alignment; the untiled form writes D, P and B)."""
    kind = case["kind"]
    d = case.get("d", 12)
    shapes = _shapes(case) if "pairs" in case else [(case["n"], case["m"])]
    frames, cells = sum(n + m for n, m in shapes), sum(n * m for n, m in shapes)
    path = 16 * frames
    if kind == "cost":
        return {"bytes": 8 * cells + path, "flops": 12 * cells}
    if kind == "untiled":
        return {"bytes": (8 + 13) * cells + path, "flops": 12 * cells}
    if kind == "train":
        px = cells / POOL ** 2
        p1, p2 = px / STRIDES[0] ** 2, px / (STRIDES[0] * STRIDES[1]) ** 2
        # forward, weight gradients of three layers, data gradients of two
        flops = 2 * d * px + 2 * 9 * 32 * (2 * p1 + 3 * 32 * p2 + 3 * p2)
        return {"bytes": 8 * d * frames + 4 * (px + 2 * 32 * (p1 + p2)), "flops": flops}
    kept = sum(n + m for n, m in shapes) * 2 * case["L"] if kind == "pruned" else cells
    return {"bytes": 8 * d * frames + path, "flops": (2 * d + 1 + 12) * kept}


# -- the same results in 64 bits, in plain numpy and torch -------------------
def _flexdtw(C):
    """D of the untiled recurrence and the best average cost of an end cell."""
    R, W = C.shape
    D = np.zeros((R, W))
    P = np.zeros((R, W), np.int64)
    D[0], D[:, 0] = C[0], C[:, 0]
    Cf, Df, Pf = C.reshape(-1), D.reshape(-1), P.reshape(-1)
    for s in range(2, R + W - 1):
        r = np.arange(max(1, s - W + 1), min(R - 1, s - 1) + 1)
        at = r * W + (s - r)
        c = s - r
        best, best_q, best_p = np.full(r.size, np.inf), np.full(r.size, np.inf), 0 * r
        for (dr, dc), w in zip(STEPS, WEIGHTS):
            ok = (r >= dr) & (c >= dc)
            pr, pc = np.where(ok, r - dr, 0), np.where(ok, c - dc, 0)
            a = Df[pr * W + pc] + Cf[at] * w
            p = np.where(pr == 0, pc, np.where(pc == 0, -pr, Pf[pr * W + pc]))
            # the start's distance: the predecessor's own code, 0 on the border
            q = np.where(ok, a / np.maximum(s - np.abs(Pf[pr * W + pc]), 1), np.inf)
            win = q < best_q
            best, best_p = np.where(win, a, best), np.where(win, p, best_p)
            best_q = np.where(win, q, best_q)
        Df[at], Pf[at] = best, best_p
    ends = [(R - 1, c) for c in range(1, W)] + [(r, W - 1) for r in range(R - 2, 0, -1)]
    return D, min(D[r, c] / (r + c - abs(P[r, c])) for r, c in ends)


def _pooled_exact(F):
    A = torch.from_numpy(F)
    A = A / A.norm(dim=0, keepdim=True)
    return torch.stack([x.mean(dim=1) for x in A.split(POOL, dim=1)], dim=1)


def _train_exact(case, seed):
    F1, F2 = _features(case, seed)
    x = 1.0 - _pooled_exact(F1).T @ _pooled_exact(F2)
    x = x - x.mean(1, keepdim=True) - x.mean(0, keepdim=True) + x.mean()
    x = (x / x.square().mean().sqrt())[None, None]
    p = {k: v.double().cpu().requires_grad_() for k, v in TileProposer(seed=seed).params.items()}
    for k, s in enumerate(STRIDES, 1):
        x = torch.nn.functional.conv2d(x, p["w%d" % k], p["b%d" % k], stride=s, padding=1)
        x = x.relu() if k < 3 else x
    x, lab, hop, fpp = x[0, 0], _labels(case), case["L"] - 1, POOL * STRIDES[0] * STRIDES[1]
    H, W = x.shape

    def span(i, size, n):
        lo, hi = i * hop, min(n, i * hop + case["L"])
        lo = min(lo // fpp, size - 1)
        return lo, max(min(-(-hi // fpp), size), lo + 1)
    score = []
    for i in range(lab.shape[0]):
        for j in range(lab.shape[1]):
            (y0, y1), (x0, x1) = span(i, H, case["n"]), span(j, W, case["m"])
            score.append(x[y0:y1, x0:x1].max())
    y = torch.from_numpy(lab.reshape(-1)).double()
    loss = torch.nn.functional.binary_cross_entropy_with_logits(
        torch.stack(score), y, pos_weight=torch.tensor(POS_WEIGHT, dtype=torch.float64))
    loss.backward()
    new = {k: (v - LR * v.grad / (v.grad.abs() + 1e-8)).detach() for k, v in p.items()}
    return {"loss": loss.detach().reshape(1), "grads": {k: v.grad for k, v in p.items()},
            "params": new}


def exact(case, seed):
    if case["kind"] == "untiled":
        D, best = _flexdtw(_cost(case, seed).cpu().numpy())
        return {"best": best, "wp": None, "D": D, "P": None, "B": None}
    if case["kind"] == "train":
        return _train_exact(case, seed)
    return None  # the tiled alignment, cell by cell in NumPy, takes minutes
