"""Workloads of the FSMELD search engine, for timing and for comparing results.

A case is one call of the public Python API (`fsmeld_b200.api`) on a target
that is already resident on the GPU, the way a program holds it: an `Engine`
over the series, the query, and the distance cutoff, which the program got
from a `cutoff` call before (the documented use: rank-k distance first, then
`search` or `exact` at it).  Targets are the seeded random walks of
`fsmeld_b200.synth` (plain; with motifs, NaN spans and flat runs; with
bursts), queries are noisy windows of them.

Fields of a case
  call     search | cutoff | exact | noalloc, or batch_search | batch_cutoff
  n        target points
  m, w     query length and band radius; a batch with m_lo has lengths
           uniform on [m_lo, m] and w = floor(0.05 m) per query
  metric   dtw | erp | edr | lcss | msm, or "all": the five in turn
  k        rank whose distance is the cutoff, or the k of `cutoff`
  queries  number of queries of a batch
  target   walk | struct | bursts
  raw      raw (non-normalised) mode
"""
import math

import numpy as np
import torch

from fsmeld_b200 import api
from fsmeld_b200.synth import query_from, random_walk, walk_with_bursts, walk_with_structure

METRICS = ("dtw", "erp", "edr", "lcss", "msm")
ARGS = {"dtw": 0.0, "erp": 0.0, "edr": 0.25, "lcss": 0.25, "msm": 0.5}
# a cutoff is the rank-k distance, raised a little so that the k-th match does
# not hang on the last bit of its distance
RAISE = 1.0 + 1e-6
# matches a program keeps of one query; their number varies with the series
# (the count says how many there were), unused entries hold -1 and 0.0
KEEP = 4096


def _case(name, call, n, m, w, metric, k, queries=1, target="walk", m_lo=0, raw=False):
    return {"name": name, "call": call, "n": n, "m": m, "w": w, "metric": metric, "k": k, "queries": queries,
            "target": target, "m_lo": m_lo, "raw": raw}


def listed():
    return [
        # the smallest request: a short recording, a short pattern; launches and host work count
        _case("search_tiny", "search", 1 << 13, 48, 4, "dtw", 5, target="struct"),
        # a small ranking on an odd length: fixing a cutoff interactively
        _case("cutoff_small", "cutoff", 65_537, 96, 6, "erp", 20),
        # the plain single search: one million points, DTW, rank-10 cutoff
        _case("search_dtw_1m", "search", 1 << 20, 128, 6, "dtw", 10),
        # the headline workload: five metrics over one 2^24-point structured series
        _case("search_five_16m", "batch_search", 1 << 24, 256, 13, "all", 50, queries=5, target="struct"),
        # a metric whose bounds prune little, odd sizes: verification work dominates
        _case("search_msm_3m", "search", 3_000_017, 391, 19, "msm", 10),
        # many patterns of one shape against one series (shared statistics and envelopes)
        _case("search_group32", "batch_search", 1 << 22, 128, 6, "dtw", 10, queries=32),
        # batched rankings on a bursty series
        _case("cutoff_group8", "batch_cutoff", 1 << 23, 512, 26, "dtw", 10, queries=8, target="bursts"),
        # a mixed queue: uneven lengths, metrics round-robin
        _case("search_mixed20", "batch_search", 1 << 22, 1024, 51, "all", 10, queries=20, m_lo=64),
        # long pattern, wide band
        _case("search_long", "search", 1 << 21, 1850, 138, "erp", 10),
        # every window through the exact distance
        _case("exact_lcss", "exact", 400_009, 160, 8, "lcss", 25),
        # the same for a caller that owns all device memory, on the caller's stream
        _case("exact_noalloc", "noalloc", 120_000, 200, 10, "dtw", 25),
        # raw values, no normalisation
        _case("search_raw", "search", (1 << 20) + 1, 250, 12, "erp", 10, raw=True),
    ]


def draw(rng):
    def log(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    call = rng.choice(("search", "search", "search", "cutoff", "cutoff", "exact", "noalloc", "batch_search",
                       "batch_cutoff"))
    metric = rng.choice(METRICS)
    m = log(32, 1500)
    w = rng.randint(0, m // 10)
    k = log(2, 100)
    queries, m_lo, raw = 1, 0, False
    target = rng.choice(("walk", "walk", "struct", "bursts"))
    if call == "search":
        n = log(1 << 13, 1 << 22)
        raw = rng.random() < 0.15
    elif call == "cutoff":
        n = log(1 << 13, 1 << 21)
    elif call in ("exact", "noalloc"):
        n, m, w = log(1 << 13, 1 << 18), min(m, 600), min(w, 30)
        target = "walk"
    else:
        n = log(1 << 16, 1 << 22)
        queries = log(2, 32)
        form = rng.choice(("same", "mixed", "all"))
        if form == "mixed":
            m, m_lo, metric = max(m, 96), 64, "all"
            w = m * 5 // 100
        elif form == "all":
            metric = "all"
    n = max(n, 10 * m)
    # no more work than the largest listed case: points x band cells of a row
    most = float(1 << 24) * 27 * 5
    while n * float(2 * w + 1) * queries * (m / 256.0) > most / 8 and n > 20 * m:
        n = int(n * 0.8)
    n += rng.randint(0, 63)
    if call == "noalloc":
        n = min(n, 262_144 + m - 1)
    return {key: v for key, v in _case("", call, n, m, w, metric, k, queries, target, m_lo, raw).items()
            if key != "name"}


def _target(case, seed):
    if case["target"] == "struct":
        return walk_with_structure(case["n"], min(case["m"], case["n"] // 64), seed=[seed, 1],
                                   motifs=max(4, min(200, case["n"] // 4096)), nan_fraction=1e-3,
                                   flat_runs=max(1, min(50, case["n"] // 65536)))
    if case["target"] == "bursts":
        return walk_with_bursts(case["n"], min(case["m"], case["n"] // 64), seed=[seed, 2])
    return random_walk(case["n"], [seed, 3])


def _inputs(case, seed):
    """The target and the queries, from the seed alone."""
    t = _target(case, seed)
    rng = np.random.default_rng([seed, 4])
    qs = []
    for i in range(case["queries"]):
        m, w = case["m"], case["w"]
        if case["m_lo"]:
            m = int(rng.integers(case["m_lo"], case["m"] + 1))
            w = m * 5 // 100
        metric = METRICS[i % 5] if case["metric"] == "all" else case["metric"]
        q, _ = query_from(t, m, rng)
        qs.append({"query": q, "m": m, "w": w, "metric": metric, "arg": ARGS[metric], "k": case["k"]})
    return t, qs


def _engine(case, target):
    e = api.Engine(target)
    if case["raw"]:
        e.set_normalization("raw")
    return e


def prepare(case, seed):
    t, qs = _inputs(case, seed)
    call = case["call"]
    e = _engine(case, t)
    if call not in ("cutoff", "batch_cutoff"):
        for d in qs:
            _, dist, _ = e.cutoff(d["query"], d["m"], case["k"], d["metric"], d["w"], d["arg"])
            d["cutoff"] = float(dist[-1]) * RAISE
    state = {"case": case, "qs": qs, "engine": e}
    if call == "noalloc":
        e.close()
        state["target"] = torch.from_numpy(t).cuda()
        state["idx"] = torch.zeros(case["n"], dtype=torch.int64, device="cuda")
        state["dist"] = torch.zeros(case["n"], dtype=torch.float64, device="cuda")
    return state


def _kept(values, fill):
    out = np.full(KEEP, fill, dtype=values.dtype)
    out[:min(KEEP, len(values))] = values[:KEEP]
    return out


def run(state):
    case, qs, e = state["case"], state["qs"], state["engine"]
    call, d = case["call"], qs[0]
    if call == "search":
        idx, c = e.search(d["query"], d["m"], d["cutoff"], d["metric"], d["w"], d["arg"])
        return {"idx": _kept(idx, -1), "counters": np.array([len(idx), c["valid"], c["after_lb"], c["after_glb"]])}
    if call == "cutoff":
        idx, dist, c = e.cutoff(d["query"], d["m"], d["k"], d["metric"], d["w"], d["arg"])
        return {"idx": idx, "dist": dist, "counters": np.array([c["valid"]])}
    if call == "exact":
        idx, dist, c = e.exact(d["query"], d["m"], d["cutoff"], d["metric"], d["w"], d["arg"])
        return {"idx": _kept(idx, -1), "dist": _kept(dist, 0.0), "counters": np.array([len(idx), c["valid"]])}
    if call == "noalloc":
        n = api.exact_noalloc(state["target"].data_ptr(), case["n"], d["query"], d["m"], d["cutoff"], d["metric"],
                              d["w"], d["arg"], state["idx"].data_ptr(), state["dist"].data_ptr(), case["n"],
                              stream=torch.cuda.current_stream().cuda_stream)
        # the caller's buffers: the first n entries are this call's
        return {"idx": state["idx"], "dist": state["dist"], "count": n}
    mode = call.split("_")[1]
    res = e.batch(mode, qs)
    if any(r["status"] for r in res):
        raise RuntimeError("a query of the batch failed")
    # queries of equal shape may share one bound per group, so only the counts
    # that do not depend on that are results
    out = {"idx": np.stack([_kept(r["idx"], -1) for r in res]),
           "counts": np.array([[r["count"], r["counters"]["valid"]] for r in res])}
    if mode == "cutoff":
        out["dist"] = np.stack([r["dist"] for r in res])
    return out


# FP64 operations per band cell of each recurrence
CELL = {"dtw": 5, "erp": 11, "edr": 8, "lcss": 6, "msm": 27}


def _segment(m, n):
    sel = 1
    while sel < 8 * m:
        sel *= 2
    return min(sel, n)


def work(case):
    """The target read once, the queries read and the results written once;
    running sums per window and, for a scan of all windows, one band row of
    each window at least (no window can be dismissed without one), else the
    lower bound's transform per macro segment; the k results' full distances."""
    flops, rows = 0.0, case["queries"]
    cells = [CELL[x] for x in (METRICS if case["metric"] == "all" else (case["metric"],))]
    cell = sum(cells) / len(cells)
    m = (case["m"] + case["m_lo"]) // 2 if case["m_lo"] else case["m"]
    w = m * 5 // 100 if case["m_lo"] else case["w"]
    lengths = rows if case["m_lo"] else 1
    flops += 12.0 * case["n"] * lengths
    if case["call"] in ("exact", "noalloc"):
        flops += rows * float(case["n"]) * (2 * w + 1) * cell
    else:
        seg = _segment(m, case["n"])
        flops += rows * (case["n"] / float(seg - m + 1)) * 15.0 * seg * math.log2(max(2, seg))
    flops += rows * float(case["k"]) * m * (2 * w + 1) * cell
    return {"bytes": 8.0 * case["n"] + rows * (8.0 * m + 16.0 * case["k"]), "flops": flops}


# ------------------------------------------------------------ in 64 bits, by plain torch

def _msm_c(new, x, y, c):
    between = ((x <= new) & (new <= y)) | ((y <= new) & (new <= x))
    return torch.where(between, torch.full_like(x, c), c + torch.minimum((new - x).abs(), (new - y).abs()))


def _distances(target, q, m, w, metric, arg, raw):
    """Banded elastic distance of every window of the target to the query."""
    t = torch.from_numpy(target).cuda()
    x = torch.from_numpy(np.asarray(q, dtype=np.float64))
    if not raw:
        x = (x - x.mean()) / x.std(unbiased=False)
    x = x.tolist()
    out = []
    for a in range(0, len(t) - m + 1, 1 << 17):
        win = t[a:a + (1 << 17) + m - 1].unfold(0, m, 1)
        ok = torch.isfinite(win).all(1)
        if raw:
            y = win.T.contiguous()
        else:
            mean = win.mean(1, keepdim=True)
            sd = ((win - mean) ** 2).mean(1, keepdim=True).sqrt()
            ok = ok & (sd[:, 0] > 1e-12)
            y = ((win - mean) / sd).T.contiguous()
        d = _band(x, y, m, w, metric, arg)
        out.append(torch.where(ok, d, torch.full_like(d, math.inf)))
    return torch.cat(out)


def _band(x, y, m, w, metric, arg):
    big = torch.full_like(y[0], 0.0 if metric == "lcss" else math.inf)
    padded = metric in ("erp", "edr")  # rows and columns 0..m, row and column 0 the empty prefix
    size = m + 1 if padded else m
    prev = {}
    for i in range(size):
        cur = {}
        for j in range(max(0, i - w), min(size - 1, i + w) + 1):
            up, left, diag = prev.get(j, big), cur.get(j - 1, big), prev.get(j - 1, big)
            if metric == "dtw":
                best = torch.zeros_like(big) if i == j == 0 else torch.minimum(torch.minimum(up, left), diag)
                cur[j] = best + (x[i] - y[j]) ** 2
            elif metric == "lcss":
                hit = (x[i] - y[j]).abs() <= arg
                cur[j] = torch.maximum(torch.maximum(up, left), torch.where(hit, diag + 1.0, diag))
            elif metric == "erp":
                if i == j == 0:
                    cur[j] = torch.zeros_like(big)
                    continue
                best = big
                if i and j:
                    best = diag + (x[i - 1] - y[j - 1]) ** 2
                if i:
                    best = torch.minimum(best, up + (x[i - 1] - arg) ** 2)
                if j:
                    best = torch.minimum(best, left + (y[j - 1] - arg) ** 2)
                cur[j] = best
            elif metric == "edr":
                if not (i and j):
                    cur[j] = torch.full_like(big, float(i + j))
                    continue
                miss = ((x[i - 1] - y[j - 1]).abs() > arg).to(big.dtype)
                cur[j] = torch.minimum(torch.minimum(up, left) + 1.0, diag + miss)
            else:
                xi = torch.full_like(big, x[i])
                if i == j == 0:
                    cur[j] = (xi - y[0]).abs()
                    continue
                best = big
                if i and j:
                    best = diag + (xi - y[j]).abs()
                if i:
                    best = torch.minimum(best, up + _msm_c(xi, torch.full_like(big, x[i - 1]), y[j], arg))
                if j:
                    best = torch.minimum(best, left + _msm_c(y[j], xi, y[j - 1], arg))
                cur[j] = best
        prev = cur
    last = prev[size - 1]
    if metric in ("dtw", "erp"):
        return last.sqrt()
    return 1.0 - last / m if metric == "lcss" else last


def exact(case, seed):
    """The distances that a call returns; a search returns whole numbers only."""
    if case["call"] not in ("cutoff", "exact", "noalloc") or case["target"] == "struct":
        return None
    steps = math.ceil(case["n"] / float(1 << 17)) * case["m"] * (2.0 * case["w"] + 1)
    if steps > 40_000:  # tens of seconds
        return None
    t, qs = _inputs(case, seed)
    d = qs[0]
    dist = _distances(t, d["query"], d["m"], d["w"], d["metric"], d["arg"], case["raw"])
    ranked = torch.sort(dist).values
    if case["call"] == "cutoff":
        return {"idx": None, "dist": ranked[:case["k"]].cpu().numpy(), "counters": None}
    value = dist[dist <= ranked[case["k"] - 1] * RAISE].cpu().numpy()
    if case["call"] == "noalloc":
        whole = np.zeros(case["n"])
        whole[:len(value)] = value
        return {"idx": None, "dist": whole, "count": None}
    return {"idx": None, "dist": _kept(value, 0.0), "counters": None}
