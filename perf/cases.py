"""What a user has this library do, as cases that can be measured: interval searches of every size the drop-in, the
batch queue and the serving loop issue, through the public entry points of the Python binding (hss.Search).

A case is a dict of plain values; `prepare` opens the handle a program keeps and picks the root intervals from the seed,
`run` makes one call (or one burst of served requests) and returns every counter the reference defines, the per-row counts
where the call gives them, and the hits.  Device times, launch counts and copied bytes differ from run to run and are not
results; neither is the number of products a build settles on its exact path, which is its own affair.
"""
import math
import random
import sys
from functools import lru_cache
from pathlib import Path

import numpy as np

sys.path.insert(0, str(Path(__file__).resolve().parents[1] / "heronian-square-search_gb300"))
import hss  # noqa: E402

COUNTERS = ("processed", "products", "candidates", "r16", "merged", "merged_products", "merged_candidates",
            "merged_r16", "hits")


def listed():
    return [
        # the smallest call: one root edge at LIMIT 70,000 (the reference's single-point smoke case), a root of one split prime
        {"name": "row_70k", "kind": "search", "limit": 70_000, "rows": 1, "at": 11_789, "spread": 2_000, "weight": 5},
        # the reference's CPU regression, root edges 1..5000 at LIMIT 5000, less a few rows at its end
        {"name": "all_5k", "kind": "search", "limit": 5_000, "rows": 4_900, "at": 1, "spread": 100, "weight": 0},
        # a contiguous sweep at LIMIT 100,000: 16,384 roots of the 1..100,000 interval, an uneven start
        {"name": "sweep_100k", "kind": "search", "limit": 100_000, "rows": 16_384, "at": 20_011, "spread": 20_000, "weight": 0},
        # one reference batch at production scale: 512 roots near 7,500,000 at LIMIT 10^7
        {"name": "batch_10m", "kind": "search", "limit": 10_000_000, "rows": 512, "at": 7_480_000, "spread": 40_000, "weight": 0},
        # the ragged end of a queue stage at LIMIT 10^7: 37 roots near 9,600,000, where windows are narrow
        {"name": "tail_10m", "kind": "search", "limit": 10_000_000, "rows": 37, "at": 9_550_001, "spread": 100_000, "weight": 0},
        # three low roots against every m up to 10^7: the longest rows there are
        {"name": "low_10m", "kind": "search", "limit": 10_000_000, "rows": 3, "at": 150_000, "spread": 200_000, "weight": 0},
        # one heavy root (branch weight 625: four split primes), as the heavy-root queue searches them
        {"name": "heavy_10m", "kind": "search", "limit": 10_000_000, "rows": 1, "at": 1_100_000, "spread": 6_000_000, "weight": 625},
        # many uneven intervals in one launch sequence under a CUDA graph, heavy starts among them
        {"name": "many_1m", "kind": "many", "limit": 1_000_000, "intervals": 24, "longest": 128},
        # a burst of requests to the serving loop: lengths log-uniform, uniform starts
        {"name": "serve_100k", "kind": "serve", "limit": 100_000, "intervals": 32, "longest": 512},
        # a caller that may not allocate while it searches: 8 roots of the production batch
        {"name": "noalloc_10m", "kind": "noalloc", "limit": 10_000_000, "rows": 8, "at": 7_480_000, "spread": 40_000, "weight": 0},
        # the plain form (the reference's launch shape), used to check the batched one
        {"name": "plain_5k", "kind": "plain", "limit": 5_000, "rows": 1_000, "at": 1, "spread": 2_000, "weight": 0},
        # the start of every worker process: the factor cache built and a first root searched
        {"name": "open_10m", "kind": "open", "limit": 10_000_000, "rows": 1, "at": 7_480_000, "spread": 40_000, "weight": 5},
    ]


def draw(rng):
    """One more case of these ranges: a kind by how often it is met, its sizes over their whole range (by their logarithm)."""
    def log_int(a, b):
        return int(round(math.exp(rng.uniform(math.log(a), math.log(b)))))

    kind = rng.choice(["search"] * 7 + ["many", "serve", "noalloc", "plain", "open"])
    # logical pairs of a pass: a third of the production batch's at most, so that heavy roots among them stay below its cost
    if kind == "many" or kind == "serve":
        limit = log_int(30_000, 1_000_000 if kind == "many" else 150_000)
        longest = log_int(8, 400)
        most = max(2, min(40, int(4e8 * math.log(longest) / (longest * limit))))
        return {"kind": kind, "limit": limit, "intervals": rng.randint(2, most), "longest": longest}
    limit = {"plain": log_int(1_000, 20_000), "open": log_int(100_000, 10_000_000), "noalloc": log_int(5_000, 10_000_000)}.get(
        kind) or log_int(2_000, 10_000_000)
    most = {"plain": 400, "open": 1, "noalloc": 64}.get(kind, 8_192)
    rows = max(1, min(log_int(1, most), int(4e8 / limit), limit // 2))
    at = rng.randint(1, max(1, limit - rows - limit // 20))
    weight = rng.choice([5, 25, 125]) if rows == 1 else 0
    return {"kind": kind, "limit": limit, "rows": rows, "at": at, "spread": max(2, limit // 25), "weight": weight}


def branch_weights(first, rows):
    """prod (4e + 1) over the primes = 1 mod 4 of every root first .. first + rows - 1."""
    x = np.arange(first, first + rows, dtype=np.int64)
    rest, w = x.copy(), np.ones(rows, dtype=np.int64)
    for p in _primes(math.isqrt(first + rows)):
        at = np.arange(-first % p, rows, p)
        e = np.zeros(len(at), dtype=np.int64)
        sub = rest[at]
        while len(sub):
            d = sub % p == 0
            if not d.any():
                break
            sub = np.where(d, sub // p, sub)
            e += d
        rest[at] = sub
        if p % 4 == 1:
            w[at] *= 4 * e + 1
    return np.where((rest > 1) & (rest % 4 == 1), w * 5, w)


@lru_cache(maxsize=None)
def _primes(n):
    s = np.ones(n + 1, dtype=bool)
    s[:2] = False
    for i in range(2, math.isqrt(n) + 1):
        if s[i]:
            s[i * i::i] = False
    return [int(p) for p in np.nonzero(s)[0]]


def _first(case, seed):
    """The case's first root for a seed.  A single root is the next one of the case's branch weight (1 taken for "any"); of an
    interval's starts, the middle one by weight of nine, so that one seed costs about what another does."""
    rng = random.Random(seed)
    limit, rows = case["limit"], case["rows"]
    top = limit - rows + 1
    if rows == 1 and case["weight"]:
        start = min(top, case["at"] + rng.randrange(case["spread"]))
        for a in [start, 1]:
            n = min(200_000, limit - a + 1)
            hit = np.nonzero(branch_weights(a, n) == case["weight"])[0]
            if len(hit):
                return a + int(hit[0])
        return start
    starts = [max(1, min(top, case["at"] + rng.randrange(case["spread"]))) for _ in range(9)]
    cost = lambda a: int(branch_weights(a, rows).sum()) * (limit - a + 1)  # noqa: E731
    return sorted(starts, key=cost)[4]


def _intervals(case, seed):
    return hss.uneven_intervals(seed, case["intervals"], case["limit"], max_len=min(case["longest"], case["limit"] // 2))


def prepare(case, seed):
    """The open handle a program keeps, and its intervals."""
    state = {"case": case, "limit": case["limit"]}
    if case["kind"] in ("many", "serve"):
        state["intervals"] = _intervals(case, seed)
    else:
        state["first"] = _first(case, seed)
        state["last"] = state["first"] + case["rows"] - 1
    if case["kind"] != "open":
        state["search"] = hss.Search(case["limit"], use_graph=1 if case["kind"] == "many" else 0)
    if case["kind"] == "serve":
        state["search"].serve_start()
    return state


def _result(counts, hits, rows=None):
    out = {"pairs": np.array([counts["pairs"]], dtype=np.int64),
           "counts": np.array([counts[k] for k in COUNTERS], dtype=np.int64),
           "hits": np.array(hits, dtype=np.int64).reshape(-1, 4)}
    if rows is not None:
        out["rows"] = np.array(rows, dtype=np.int64)
    return out


def run(state):
    kind = state["case"]["kind"]
    if kind in ("search", "plain"):
        r = state["search"].search(state["first"], state["last"], mode="plain" if kind == "plain" else "batched", rows=True)
        return _result(r.counts, r.hits, r.row_candidates)
    if kind == "noalloc":
        r = state["search"].search_noalloc(state["first"], state["last"])
        return _result(r.counts, r.hits)
    if kind == "many":
        per, total = state["search"].search_many(state["intervals"])
        return {**_result(total.counts, total.hits), "each": np.array([[p[k] for k in ("pairs",) + COUNTERS] for p in per], dtype=np.int64)}
    if kind == "serve":
        s = state["search"]
        done = [s.wait(i) for i in [s.submit(a, b) for a, b in state["intervals"]]]
        return {"each": np.array([[d["counts"][k] for k in ("pairs",) + COUNTERS] for d in done], dtype=np.int64),
                "hits": np.array([h for d in done for h in d["hits"]], dtype=np.int64).reshape(-1, 4)}
    with hss.Search(state["limit"]) as s:
        info = s.info()
        r = s.search(state["first"], state["last"], rows=True)
        return {**_result(r.counts, r.hits, r.row_candidates),
                "info": np.array([info[k] for k in ("limit", "records", "flattened", "cached")], dtype=np.int64)}


@lru_cache(maxsize=4)
def _weights_sum(limit):
    """sum of branch weights over 1 .. x for every x <= limit (each root's Gaussian products are about half its weight times m's)."""
    w = np.ones(limit + 1, dtype=np.int32)
    small = np.array(_primes(limit), dtype=np.int64)
    for p in small[small % 4 == 1].tolist():
        q, e = p, 1
        while q <= limit:
            w[q::q] = w[q::q] // (4 * e - 3) * (4 * e + 1)
            q, e = q * p, e + 1
    w[0] = 0
    return np.cumsum(w, dtype=np.float64)


def work(case):
    """Bytes: each 16-byte value of the roots m once (half of m's branch weight), one counter per row out.  Operations: two
    multiply-adds for each product whose real part can lie inside the window (about 0.35 of the products of the pairs that
    are not skipped, which are about 0.64 of all)."""
    limit = case["limit"]
    total = _weights_sum(limit)
    spans = [(a, b) for a, b in _intervals(case, 1)] if "intervals" in case else [(_first(case, 1),) * 2]
    if "rows" in case:
        spans = [(spans[0][0], spans[0][0] + case["rows"] - 1)]
    products, low = 0.0, min(a for a, _ in spans)
    for a, b in spans:
        w = branch_weights(a, b - a + 1).astype(np.float64)
        products += float((w * (total[limit] - total[np.arange(a, b + 1) - 1])).sum()) / 2
    records = (total[limit] - (0 if case["kind"] == "open" else total[low - 1])) / 2
    rows = sum(b - a + 1 for a, b in spans)
    return {"bytes": 16.0 * records * (2 if case["kind"] == "open" else 1) + 8.0 * rows, "flops": 4 * 0.35 * 0.64 * products}


def exact(case, seed):
    """Every output is a whole number, held equal; of them only the logical pairs have a closed form."""
    if "intervals" in case:
        return None
    first, last = _first(case, seed), _first(case, seed) + case["rows"] - 1
    pairs = sum(case["limit"] - l + 1 for l in range(first, last + 1))
    return {"pairs": np.array([pairs], dtype=np.int64), "counts": None, "hits": None, "rows": None, "info": None}
