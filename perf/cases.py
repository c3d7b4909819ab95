"""Timed cases of the library, each one call (or one short search) through the public entry points.

The sizes are those of this repository's benchmark, tests and drivers: 64 sets of k = 8, 10,000 sets
of |P| ~ U{6..14}, 2,000 sets of k = 15 with an early-exit threshold, 1,000,000 masks of popcount
5..30, driver batches of 50,000 sets, and the search levels of the canonical BFS.

  one        max_zeros of a single set: a driver rechecks one candidate exactly and waits for the
             answer, so launches and round trips count
  batch      max_zeros_batch of many sets at td = 1 (every value exact): the batched evaluation of
             a search level, uniform or of mixed k
  threshold  max_zeros_batch with a target distance per set: a generation of an evolutionary search,
             where most sets fail early against the best-known distance of their k
  screen     max_zeros_batch with sample_count: the screening of sets too large to enumerate
  keys       CanonicalOracle.compute: packed canonical keys of equal-size rows (a driver's chunk)
  masks      compute_masks of masks of any size, then CanonicalDedup: symmetry reduction of a pool
  level      CanonicalBFS.level: one level of the canonical search from n surviving parents (expand,
             canonicalise, dedup, compact, evaluate)

The device-resident request loop and the micro-batch server answer an equivalent request from what
they answered before, so passes over the same requests would time that table; their evaluation is
the walk of the cases here.

All results are whole numbers, and where the contract leaves a value open (a set that fails its
threshold reports some witness above 49 - td) `run` returns the decision in its place.
"""

from __future__ import annotations

import random

import numpy as np
import torch

from generalized_toric_gpu_search_b200 import (
    CanonicalBFS,
    CanonicalDedup,
    CanonicalOracle,
    DistanceOracleCUDABP,
    build_eval_matrix,
)

# Best-known distances a search holds as thresholds (the benchmark's table; below k = 12 the
# distances that a search of this length reaches).
BEST_D = {6: 33, 7: 33, 8: 32, 9: 30, 10: 29, 11: 28, 12: 28, 13: 27, 14: 26, 15: 24}


def listed():
    return [
        # recheck of one candidate: a small code, and the largest of the batched workload
        {"name": "one_k8", "kind": "one", "k_lo": 8, "k_hi": 8, "n": 1},
        {"name": "one_k14", "kind": "one", "k_lo": 14, "k_hi": 14, "n": 1},
        # the plain configuration: a small uniform batch
        {"name": "batch_64_k8", "kind": "batch", "k_lo": 8, "k_hi": 8, "n": 64},
        # one generation of mutated children with running best-known thresholds
        {"name": "threshold_257_k10_15", "kind": "threshold", "k_lo": 10, "k_hi": 15, "n": 257},
        # the headline workload: an uneven batch, no threshold
        {"name": "batch_10000_k6_14", "kind": "batch", "k_lo": 6, "k_hi": 14, "n": 10000},
        # high k with an early-exit threshold
        {"name": "threshold_2000_k15", "kind": "threshold", "k_lo": 15, "k_hi": 15, "n": 2000},
        # exact verification of large candidates
        {"name": "batch_50_k16_18", "kind": "batch", "k_lo": 16, "k_hi": 18, "n": 50},
        # sampled screening of a level of large sets
        {"name": "screen_2000_k16_30", "kind": "screen", "k_lo": 16, "k_hi": 30, "n": 2000,
         "samples": 3000},
        # a driver's canonicalisation chunk
        {"name": "keys_50000_k9", "kind": "keys", "k_lo": 9, "k_hi": 9, "n": 50000},
        # canonical masks and dedup of a large pool
        {"name": "masks_1000000", "kind": "masks", "k_lo": 5, "k_hi": 30, "n": 1000000},
        # one level of a pruned canonical search
        {"name": "level_1000_k10", "kind": "level", "k_lo": 10, "k_hi": 10, "n": 1000},
    ]


def _log_int(rng, lo, hi):
    return int(round(lo * (hi / lo) ** rng.random()))


def draw(rng):
    kind = rng.choice(["one", "batch", "batch", "batch", "threshold", "threshold", "screen", "keys",
                       "masks", "level"])
    if kind == "one":
        k = rng.randint(2, 15)
        return {"kind": kind, "k_lo": k, "k_hi": k, "n": 1}
    if kind == "batch":
        if rng.random() < 0.3:  # a few large sets
            lo = rng.randint(15, 18)
            hi = rng.randint(lo, 18)
            return {"kind": kind, "k_lo": lo, "k_hi": hi, "n": _log_int(rng, 2, 50)}
        lo = rng.randint(2, 14)
        hi = rng.randint(lo, 14)
        return {"kind": kind, "k_lo": lo, "k_hi": hi, "n": _log_int(rng, 2, 10000)}
    if kind == "threshold":
        lo = rng.randint(6, 15)
        hi = rng.randint(lo, 15)
        return {"kind": kind, "k_lo": lo, "k_hi": hi, "n": _log_int(rng, 16, 4000)}
    if kind == "screen":
        lo = rng.randint(10, 40)
        hi = rng.randint(lo, 40)
        return {"kind": kind, "k_lo": lo, "k_hi": hi, "n": _log_int(rng, 16, 3000),
                "samples": _log_int(rng, 500, 4000)}
    if kind == "keys":
        k = rng.randint(2, 10)
        return {"kind": kind, "k_lo": k, "k_hi": k, "n": _log_int(rng, 50, 100000)}
    if kind == "masks":
        lo = rng.randint(1, 20)
        hi = rng.randint(lo, 40)
        return {"kind": kind, "k_lo": lo, "k_hi": hi, "n": _log_int(rng, 100, 500000)}
    k = rng.randint(4, 11)
    return {"kind": kind, "k_lo": k, "k_hi": k, "n": _log_int(rng, 2, 1000)}


def _sets(case, seed):
    """n sorted index lists, |P| uniform in k_lo..k_hi."""
    rng = random.Random(seed)
    return [sorted(rng.sample(range(49), rng.randint(case["k_lo"], case["k_hi"])))
            for _ in range(case["n"])]


def _children(case, seed):
    """Single-point mutations of a few parents, the sizes kept in k_lo..k_hi."""
    rng = random.Random(seed)
    lo, hi = case["k_lo"], case["k_hi"]
    parents = [rng.sample(range(49), rng.randint(lo, hi)) for _ in range(max(1, case["n"] // 8))]
    out = []
    for _ in range(case["n"]):
        p = list(rng.choice(parents))
        free = [x for x in range(49) if x not in p]
        op = rng.randrange(3)
        if op == 0 and len(p) < hi:
            p.append(rng.choice(free))
        elif op == 1 and len(p) > lo:
            p.pop(rng.randrange(len(p)))
        else:
            p[rng.randrange(len(p))] = rng.choice(free)
        out.append(sorted(p))
    return out


def _masks(n, lo, hi, seed):
    """n random 49-bit masks, popcount uniform in lo..hi."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    keys = torch.rand((n, 49), generator=g, device="cuda")
    pop = torch.randint(lo, hi + 1, (n, 1), generator=g, device="cuda")
    rank = torch.argsort(torch.argsort(keys, dim=1), dim=1)
    weights = torch.ones((), dtype=torch.int64, device="cuda") << torch.arange(49, device="cuda")
    masks = ((rank < pop).to(torch.int64) * weights).sum(dim=1)
    return masks.cpu().numpy().view(np.uint64)


def prepare(case, seed):
    kind = case["kind"]
    state = {"case": case}
    if kind in ("one", "batch", "threshold", "screen"):
        state["oracle"] = DistanceOracleCUDABP(0, build_eval_matrix())
        if kind == "threshold":
            state["sets"] = _children(case, seed)
            state["td"] = np.array([BEST_D[len(s)] for s in state["sets"]], dtype=np.int32)
        else:
            state["sets"] = _sets(case, seed)
        state["points"] = np.array([sum(1 << i for i in s) for s in state["sets"]])
    elif kind == "keys":
        state["oracle"] = CanonicalOracle(0)
        rng = np.random.default_rng(seed)
        rows = np.argpartition(rng.random((case["n"], 49)), case["k_lo"], axis=1)[:, :case["k_lo"]]
        state["rows"] = np.sort(rows, axis=1).astype(np.int32)
    elif kind == "masks":
        state["oracle"] = CanonicalOracle(0)
        state["dedup"] = CanonicalDedup(0, 4 * case["n"])
        state["masks"] = _masks(case["n"], case["k_lo"], case["k_hi"], seed)
    else:
        state["bfs"] = CanonicalBFS(0, dedup_capacity=1 << 20)
        k = case["k_hi"]
        parents = CanonicalOracle(0).compute_masks(_masks(case["n"], k - 1, k - 1, seed))
        state["parents"] = torch.from_numpy(np.unique(parents).view(np.int64)).cuda()
    return state


def run(state):
    case = state["case"]
    kind = case["kind"]
    # a driver records each value with its set (here as a mask)
    if kind == "one":
        return state["oracle"].max_zeros(state["sets"][0], 1), state["points"]
    if kind == "batch":
        return np.array(state["oracle"].max_zeros_batch(state["sets"], 1)), state["points"]
    if kind == "threshold":
        mz = np.array(state["oracle"].max_zeros_batch(state["sets"], state["td"]))
        # exact where the set passes, else the decision
        return np.minimum(mz, 50 - state["td"]), state["points"]
    if kind == "screen":
        return np.array(state["oracle"].max_zeros_batch(state["sets"], 1,
                                                        sample_count=case["samples"],
                                                        sample_seed=7)), state["points"]
    if kind == "keys":
        return state["oracle"].compute(state["rows"]).astype(np.int64)
    if kind == "masks":
        masks = state["oracle"].compute_masks(state["masks"])
        state["dedup"].clear()
        return masks.view(np.int64), state["dedup"].insert(masks)
    bfs = state["bfs"]
    bfs.dedup.clear(bfs.stream)
    lv = bfs.level(state["parents"], case["k_hi"], 1)
    # the classes found, one row each, in a table with room for every child
    table = torch.zeros((case["n"] * 49, 2 + case["k_hi"]), dtype=torch.int64, device="cuda")
    rows = torch.cat((lv.masks[:, None], lv.max_zeros[:, None], lv.sets), dim=1)
    table[:rows.shape[0]] = rows
    return table


def work(case):
    """Inputs read once and outputs written once.  The number of codewords, images or samples that
    the answer needs depends on the method; counted are the operations no method goes without: one
    elimination of each code's k x 49 matrix over three bit planes, one sample's k row additions,
    and one look at each point of a set per linear map."""
    n, k = case["n"], (case["k_lo"] + case["k_hi"]) / 2
    kind = case["kind"]
    if kind in ("one", "batch", "threshold"):
        return {"bytes": n * (4 * k + 8 + 4), "flops": n * 3 * 49 * k * k}
    if kind == "screen":
        return {"bytes": n * (4 * k + 8 + 4), "flops": n * case["samples"] * 3.0 * 49 * k}
    if kind == "keys":
        return {"bytes": n * (4 * k + 16), "flops": n * 2016.0 * k}
    if kind == "masks":
        return {"bytes": n * (8 + 8 + 1), "flops": n * 2016.0 * k}
    kids = n * (49 - case["k_hi"])
    return {"bytes": 8 * n + kids * (8 + 4 * k + 4), "flops": kids * (2016.0 * k + 3 * 49 * k * k)}


def exact(case, seed):
    """Every output is a whole number, which has to be the same; none is a rounded value."""
    return None
