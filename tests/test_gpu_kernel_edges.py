"""Kernels at the edges of their tiles, against the oracle (needs a B200):
lengths around the tile widths, macro segments clipped to the target, odd
segment counts, non-finite points on tile borders.  Window statistics,
envelopes, thresholds and distances are compared bit for bit."""
import numpy as np
import pytest

from fsmeld_b200.synth import query_from, random_walk
from tests.test_gpu_parity import _geom, _segments, api, bits_equal  # noqa: F401

pytestmark = pytest.mark.gpu


def _target(n, seed, bad):
    t = random_walk(n, seed)
    t[[i for i in bad if i < n]] = np.nan
    return t


# k_mvmean: tiles of 32 points, 2..16 segments a block; m around the tile
# width, m_k = n (not a multiple of 32), one segment, many segments
@pytest.mark.parametrize("n,m", [(2000, 31), (2001, 32), (5003, 33), (301, 64), (191, 96), (1 << 15, 2), (1 << 17, 5),
                                 (70_001, 129)])
def test_window_stats_tiles(api, oracle, n, m):  # noqa: F811
    t = _target(n, 5, bad=[31, 32, 63, 64 + m, 95, 1024, 1055, n - 1])
    q = random_walk(m, 6)
    segs, mk, kml = _segments(t, m)
    with api.Engine(t) as e:
        mu = e.inspect(q, m, "dtw", 0, 0.0, 0).reshape(-1, kml)
        sg = e.inspect(q, m, "dtw", 0, 0.0, 1).reshape(-1, kml)
    for s, ts in enumerate(segs):
        omu, osg = oracle.mvmean(ts, m)
        assert bits_equal(mu[s], omu), s
        assert bits_equal(sg[s], osg), s


# k_bitdp (EDR, LCSS): band widths around the word borders (2w+1 bits in 1..16
# words), lengths not a multiple of the four points of a step, ties (integer
# targets), tolerances that match nothing, little and everything
@pytest.mark.parametrize("m,w", [(2, 0), (3, 2), (33, 15), (34, 16), (66, 31), (65, 32), (101, 47), (130, 64),
                                 (299, 255)])
@pytest.mark.parametrize("metric", ["edr", "lcss"])
def test_bit_vector_distances(api, oracle, metric, m, w):  # noqa: F811
    t = random_walk(3 * m + 200, [7, m])
    t[m:2 * m] = np.round(t[m:2 * m])
    q, _ = query_from(t, m, np.random.default_rng([8, m]))
    with api.Engine(t) as e:
        for arg in (0.0, 0.25, 1.7, 1e300):
            gi, gd, gc = e.exact(q, m, 1e300, metric, w, arg)
            oi, od, oc = oracle.exact(t, q, m, 1e300, metric, w, arg)
            assert list(gi) == list(oi) and gc["valid"] == oc["valid"]
            assert bits_equal(gd, od), arg
            k = min(9, len(oi))
            ci, cd, _ = e.cutoff(q, m, k, metric, w, arg)
            xi, xd, _ = oracle.cutoff(t, q, m, k, metric, w, arg)
            assert list(ci) == list(xi) and bits_equal(cd, xd), arg
            si, sc = e.search(q, m, float(xd[-1]), metric, w, arg)
            yi, yc = oracle.search(t, q, m, float(xd[-1]), metric, w, arg)
            assert list(si) == list(yi) and sc["after_glb"] == yc["after_glb"], arg


# k_screen (DTW, ERP, MSM): odd and even row counts, narrow and wide bands (one,
# two and four warps a block), cutoffs equal to a distance, between two, below
# all; lists long enough to be screened (over 32 per SM); raw mode with large
# values; points beyond the bound's limit.  Every decision is the oracle's.
@pytest.mark.parametrize("m,w,raw", [(3, 2, False), (16, 2, False), (17, 3, False), (40, 39, False), (63, 15, False),
                                     (64, 16, True), (90, 70, False), (150, 140, False)])
@pytest.mark.parametrize("metric,arg", [("dtw", 0.0), ("erp", 0.0), ("erp", 0.4), ("msm", 0.5)])
def test_screened_distances(api, oracle, metric, arg, m, w, raw):  # noqa: F811
    n = 6000 + m
    t = random_walk(n, [9, m])
    t[2000:2010] += 500.0  # spikes: normalised points near sqrt(m)
    t[4000] = np.nan
    if raw:
        t = t * 50.0 + 1e4
    q, _ = query_from(t, m, np.random.default_rng([10, m]))
    try:
        oracle.set_normalization("raw" if raw else "zscore")
        with api.Engine(t) as e:
            e.set_normalization("raw" if raw else "zscore")
            oi, od, oc = oracle.exact(t, q, m, 1e300, metric, w, arg)
            ranked = np.sort(od)
            for cut in (ranked[0], ranked[20], 0.5 * (ranked[50] + ranked[51]), ranked[len(ranked) // 2],
                        ranked[-1], 0.5 * ranked[0]):
                keep = od <= cut
                gi, gd, gc = e.exact(q, m, float(cut), metric, w, arg)
                assert list(gi) == list(oi[keep]) and gc["valid"] == oc["valid"], cut
                assert bits_equal(gd, od[keep]), cut
                si, sc = e.search(q, m, float(cut), metric, w, arg)
                yi, yc = oracle.search(t, q, m, float(cut), metric, w, arg)
                assert list(si) == list(yi) and sc["after_glb"] == yc["after_glb"], cut
    finally:
        oracle.set_normalization("zscore")


# k_threshold: every block shape; values spread (bucket sort) and bunched by a
# spike (merge sort), runs of equal values, NaN in the envelope core
@pytest.mark.parametrize("m", [8, 32, 100, 200, 300, 800, 1500])
@pytest.mark.parametrize("metric,arg", [("dtw", 0.0), ("erp", 0.4), ("msm", 0.5), ("lcss", 0.25)])
def test_threshold_shapes(api, oracle, metric, arg, m):  # noqa: F811
    w = m // 20
    mk, kml, _, _ = _geom(m, 1 << 30)
    t = random_walk(3 * kml + m + 7, [11, m])
    t[kml + mk // 2] += 1e7                               # second segment: one far value
    t[2 * kml + mk // 2: 2 * kml + mk // 2 + mk // 4] = 3.0  # third: a flat run
    t[2 * kml + mk // 3] = np.nan
    q, _ = query_from(t[:kml], m, np.random.default_rng([12, m]))
    qn = oracle.normalize_query(q)
    with api.Engine(t) as e:
        thr = e.inspect(q, m, metric, w, arg, 4).reshape(-1, 2)
        un = e.inspect(q, m, metric, w, arg, 2).reshape(-1, mk)
        ln = e.inspect(q, m, metric, w, arg, 3).reshape(-1, mk)
    for s in range(len(thr)):
        tl = oracle.find_t(0, metric, ln[s], qn, m, arg)
        tu = oracle.find_t(1, metric, un[s], qn, m, arg)
        assert bits_equal(thr[s], [tl, tu]), (s, thr[s], tl, tu)


# k_envelope: windows read point by point (m <= 16) and by runs of eight, tiles
# of 512, 1024 and 2048 outputs with a remainder, clipped segments, NaN at the
# start, inside and at the end of windows and runs
@pytest.mark.parametrize("n,m,w", [(4000, 2, 0), (4000, 9, 8), (5000, 16, 3), (5001, 17, 1), (5002, 24, 5),
                                   (5003, 25, 24), (20_000, 100, 9), (9000, 257, 40), (90_000, 600, 30),
                                   (4300, 1500, 200), (16_001, 8000, 50)])
def test_envelope_tiles(api, oracle, n, m, w):  # noqa: F811
    for bad in ([], [7, 8, 1023, 1024 + m, n // 2, n // 2 + 1, n - 1]):
        t = _target(n, [13, m], bad)
        q = random_walk(m, 14)
        segs, mk, kml = _segments(t, m)
        with api.Engine(t) as e:
            un = e.inspect(q, m, "dtw", w, 0.0, 2).reshape(-1, mk)
            ln = e.inspect(q, m, "dtw", w, 0.0, 3).reshape(-1, mk)
        for s, ts in enumerate(segs):
            omu, osg = oracle.mvmean(ts, m)
            mn, mx = oracle.min_max_window(omu, mk, m)
            smn, smx = oracle.min_max_window(osg, mk, m)
            L, U = oracle.lemire(ts, w)
            oun, oln = oracle.normalized(U, L, mx, mn, smx, smn)
            assert bits_equal(un[s], oun), (s, len(bad))
            assert bits_equal(ln[s], oln), (s, len(bad))


# k_lbip_runs: sums over mask changes and popcounts, word borders of the masks,
# walks (few changes) and noise (many), the tail segment; the same tolerance as
# the transform's (1e-9 absolute, 1e-12 relative, squared domain for DTW, ERP).
# Narrow bands (100 (w+1) < m) keep the transform.
@pytest.mark.parametrize("m,w", [(2, 0), (31, 1), (64, 2), (65, 10), (200, 1), (300, 2), (600, 30)])
@pytest.mark.parametrize("metric,arg", [("dtw", 0.0), ("erp", 0.4), ("edr", 0.25), ("lcss", 0.25), ("msm", 0.5)])
def test_lbip_runs(api, oracle, metric, arg, m, w):  # noqa: F811
    mk, kml, _, _ = _geom(m, 1 << 30)
    t = random_walk(2 * kml + m + 5, [15, m])
    t[kml:kml + mk // 2] += np.random.default_rng([16, m]).normal(0.0, 5.0, mk // 2)
    q, _ = query_from(t, m, np.random.default_rng([17, m]))
    qn = oracle.normalize_query(q)
    with api.Engine(t) as e:
        z = e.inspect(q, m, metric, w, arg, 5).reshape(-1, kml)
        thr = e.inspect(q, m, metric, w, arg, 4).reshape(-1, 2)
        un = e.inspect(q, m, metric, w, arg, 2).reshape(-1, mk)
        ln = e.inspect(q, m, metric, w, arg, 3).reshape(-1, mk)
    _, _, forsize, tail = _geom(m, len(t))
    for s in range(len(z)):
        ref = np.correlate(oracle.s_to_g(0, ln[s], thr[s, 0]), oracle.q_to_h(0, metric, qn, thr[s, 0], arg), "valid")
        ref = ref + np.correlate(oracle.s_to_g(1, un[s], thr[s, 1]), oracle.q_to_h(1, metric, qn, thr[s, 1], arg),
                                 "valid")
        got = z[s] ** 2 if metric in ("dtw", "erp") else z[s] * m if metric == "lcss" else z[s]
        ok = ~np.isnan(got)
        if s == forsize:  # the tail segment's windows before the tail belong to other segments
            ok[:kml - tail] = False
        assert ok.sum() > 0
        assert np.all(np.abs(got - ref)[ok] <= 1e-9 + 1e-12 * np.abs(ref[ok])), s


# fsmeld_exact_noalloc: each DP it may take (screen + wavefront, bit vectors,
# lane DP for w < 2 and unreachable cutoffs), few and many matches (one block's
# order, marking and compaction), a buffer that is too small
@pytest.mark.parametrize("metric,arg", [("dtw", 0.0), ("erp", 0.4), ("msm", 0.5), ("edr", 0.25), ("lcss", 0.25)])
@pytest.mark.parametrize("m,w", [(24, 0), (24, 3), (65, 40), (2048, 20)])
def test_noalloc_paths(api, oracle, metric, arg, m, w):  # noqa: F811
    import torch

    n = 7000 + m if m < 100 else 2 * m + 300
    t = random_walk(n, [18, m])
    t[100] = np.nan
    q, _ = query_from(t, m, np.random.default_rng([19, m]))
    oi, od, _ = oracle.exact(t, q, m, 1e300, metric, w, arg)
    ranked = np.sort(od)
    d_t = torch.from_numpy(t).cuda()
    idx = torch.full((n,), -7, dtype=torch.int64, device="cuda")
    dist = torch.full((n,), -7.0, dtype=torch.float64, device="cuda")
    for cut, cap in ((ranked[10], n), (ranked[-1], n), (1e300, n), (ranked[10], 4), (ranked[-1], 5000)):
        keep = od <= cut
        c = api.exact_noalloc(d_t.data_ptr(), n, q, m, float(cut), metric, w, arg, idx.data_ptr(), dist.data_ptr(), cap)
        assert c == keep.sum()
        k = min(c, cap)
        assert np.array_equal(idx[:k].cpu().numpy(), oi[keep][:k])
        assert bits_equal(dist[:k].cpu().numpy(), od[keep][:k])


# k_lbgemm: 16 .. 128 operand columns (4 to 1 tiles at a time), the penalty
# operand resident or by chunks, lengths off the 64-element chunks, exclusions.
# A query's accumulators see the same terms in the same order in every group
# that starts with the same query (which picks the thresholds), so its survivor
# and valid counts do not depend on the group; matches are the per-query path's.
@pytest.mark.parametrize("m,w", [(33, 2), (64, 3), (129, 6), (300, 15), (700, 30)])
def test_lbgemm_groups(api, m, w):  # noqa: F811
    _, kml, _, _ = _geom(m, 1 << 30)
    t = random_walk(3 * kml + m + 77, [20, m])
    t[kml + 50] = np.nan
    rng = np.random.default_rng([21, m])
    batch = []
    for i in range(70):
        q, _ = query_from(t, m, rng)
        batch.append(dict(query=q, m=m, metric="dtw", w=w, arg=0.0, cutoff=0.2 * m ** 0.5))
    batch[2]["exclude"] = (kml - 40, kml + 300)
    with api.Engine(t) as e:
        e.set_lb_form("fft")
        ref = e.batch("search", batch)
        e.set_lb_form("gemm")
        groups = [e.batch("search", batch[:k]) for k in (3, 17, 40, 70)]
    for got in groups:
        for g, full, r in zip(got, groups[-1], ref):
            assert g["status"] == 0
            assert np.array_equal(g["idx"], r["idx"])
            assert g["counters"]["valid"] == r["counters"]["valid"]
            assert g["counters"]["matches"] == r["counters"]["matches"]
            assert g["counters"]["after_lb"] == full["counters"]["after_lb"] >= r["counters"]["matches"]


# GLB on FP32 rows (2^18 points and more): segments whose range dwarfs the
# windows' sigma (FP64 points there), flat stretches, non-finite points, windows
# without interior points, lists short enough for 8 lanes a candidate and longer
# ones; the survivor counts are the oracle's
@pytest.mark.parametrize("m,w,raw", [(24, 0, False), (33, 2, False), (40, 19, False), (130, 6, False), (24, 2, True)])
@pytest.mark.parametrize("metric,arg", [("dtw", 0.0), ("erp", 0.4), ("edr", 0.25), ("lcss", 0.25), ("msm", 0.5)])
def test_glb_fp32_rows(api, oracle, metric, arg, m, w, raw):  # noqa: F811
    n = (1 << 18) + 77
    t = random_walk(n, [22, m])
    t[5000:5300] *= 1e4
    t[9000:9400] = t[9000]
    t[12_000:14_000] = t[12_000] + 1e-3 * np.random.default_rng(3).normal(size=2000)
    t[13_000] += 1e6
    t[[100, 20_000, n - 50]] = [np.nan, np.inf, np.nan]
    q, _ = query_from(t[30_000:60_000], m, np.random.default_rng([23, m]))
    mode = "raw" if raw else "zscore"
    oracle.set_normalization(mode)
    try:
        with api.Engine(t) as e:
            e.set_normalization(mode)
            _, d, _ = e.cutoff(q, m, 20, metric, w, arg)
            for cut in (float(d[-1]) * 1.001, float(d[-1]) * 1.6):
                idx, c = e.search(q, m, cut, metric, w, arg)
                oidx, oc = oracle.search(t, q, m, cut, metric, w, arg)
                assert list(idx) == list(oidx)
                assert c["after_lb"] == oc["after_lb"]
                assert c["after_glb"] == oc["after_glb"]
    finally:
        oracle.set_normalization("zscore")


# k_screen, MSM: the first pass without intervals (a step's cost of at least
# twice the mean step of the query: here for the larger costs) and the second
# pass alone, zero cost, smooth and jumpy targets; every decision is the oracle's
@pytest.mark.parametrize("m,w", [(16, 2), (41, 6), (96, 40), (150, 8)])
@pytest.mark.parametrize("arg", [0.0, 0.05, 0.6, 2.0, 40.0])
def test_screen_msm_costs(api, oracle, arg, m, w):  # noqa: F811
    n = 5800 + m
    t = random_walk(n, [24, m])
    t[3000:4500] += np.random.default_rng([25, m]).normal(0.0, 20.0, 1500)
    t[2000:2010] += 500.0
    q, _ = query_from(t, m, np.random.default_rng([26, m]))
    oi, od, _ = oracle.exact(t, q, m, 1e300, "msm", w, arg)
    ranked = np.sort(od)
    with api.Engine(t) as e:
        for cut in (ranked[20], 0.5 * (ranked[200] + ranked[201]), ranked[len(ranked) // 2], ranked[-1]):
            keep = od <= cut
            gi, gd, _ = e.exact(q, m, float(cut), "msm", w, arg)
            assert list(gi) == list(oi[keep]), cut
            assert bits_equal(gd, od[keep]), cut


# k_screen's rows a pass (2, 4, 8 by metric and band): band widths on both sides
# of each rule, every remainder of the row count; every decision is the oracle's
@pytest.mark.parametrize("m", [25, 26, 27, 28, 29, 30, 31, 32])
@pytest.mark.parametrize("w", [3, 4, 11, 12, 24])
@pytest.mark.parametrize("metric,arg", [("dtw", 0.0), ("erp", 0.4), ("msm", 0.5)])
def test_screen_rows_a_pass(api, oracle, metric, arg, m, w):  # noqa: F811
    n = 5700 + m
    t = random_walk(n, [27, m])
    t[4100] = np.nan
    q, _ = query_from(t, m, np.random.default_rng([28, m]))
    oi, od, _ = oracle.exact(t, q, m, 1e300, metric, w, arg)
    ranked = np.sort(od)
    with api.Engine(t) as e:
        for cut in (ranked[20], 0.5 * (ranked[300] + ranked[301]), ranked[len(ranked) // 2]):
            keep = od <= cut
            gi, gd, _ = e.exact(q, m, float(cut), metric, w, arg)
            assert list(gi) == list(oi[keep]), cut
            assert bits_equal(gd, od[keep]), cut
