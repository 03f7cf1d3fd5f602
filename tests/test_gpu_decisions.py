"""Pruning decisions that hang on a single point or on the last bit of a
distance, against the oracle (needs a B200)."""
import numpy as np
import pytest

from fsmeld_b200.synth import query_from, random_walk, walk_with_structure
from tests.test_gpu_parity import api, bits_equal  # noqa: F401

pytestmark = pytest.mark.gpu


# GLB in raw mode: a window that matches but for one point far outside the
# fixed-point range (the first, the last, one inside).  The spikes' fixed-point
# words are NaN, negative and tiny floats; below 2^18 points the sums run on FP64
# points, above on FP32 rows where a segment's range allows it.
@pytest.mark.parametrize("n,spike", [(6000, 1e4), (6000, -1e4), (6000, 3e4), (6000, 1e5), (6000, 1e6), (6000, -1e6),
                                     (6000, 1e12), ((1 << 18) + 500, 1e6), ((1 << 18) + 500, 1e12)])
@pytest.mark.parametrize("metric,arg,w", [("edr", 0.25, 10), ("lcss", 0.25, 10), ("erp", 0.0, 10), ("erp", 40.0, 3),
                                          ("dtw", 0.0, 10), ("msm", 0.5, 10)])
def test_one_point_out_of_range(api, oracle, metric, arg, w, spike, n):  # noqa: F811
    m = 64
    rng = np.random.default_rng(41)
    q = np.arange(m - 1.0, -1.0, -1.0)
    t = 500.0 + rng.normal(0.0, 1.0, n)
    starts = (1000, 2000, 3000, 4000)
    for s, p in zip(starts, (0, m - 1, m // 2, 5)):
        t[s:s + m] = q - 2.0
        t[s + p] = spike
    oracle.set_normalization("raw")
    try:
        d = min(oracle.distance(metric, q, t[s:s + m].copy(), w, arg) for s in starts)
        far = max(oracle.distance(metric, q, t[s:s + m].copy(), w, arg) for s in starts)
        with api.Engine(t) as e:
            e.set_normalization("raw")
            for cut in (d, 1.5 * d, far):
                idx, c = e.search(q, m, cut, metric, w, arg)
                oidx, oc = oracle.search(t, q, m, cut, metric, w, arg)
                assert list(idx) == list(oidx), cut
                assert c["after_glb"] == oc["after_glb"], cut
            ci, cd, _ = e.cutoff(q, m, 4, metric, w, arg)
            oi, od, _ = oracle.cutoff(t, q, m, 4, metric, w, arg)
            assert list(ci) == list(oi) and bits_equal(cd, od)
    finally:
        oracle.set_normalization("zscore")


# Top-k where GLB equals the distance in exact arithmetic and exceeds it by its
# rounding: bands of radius 0 (the envelopes are the points), and flat runs beside
# each other in raw mode (many windows at the k-th distance).
@pytest.mark.parametrize("seed", range(6))
@pytest.mark.parametrize("metric,arg", [("dtw", 0.0), ("erp", 0.4), ("msm", 0.5), ("edr", 0.25), ("lcss", 0.25)])
def test_ranking_at_equal_bounds(api, oracle, metric, arg, seed):  # noqa: F811
    m = (17, 38, 40, 64, 101, 200)[seed]
    t = random_walk(5000 + m, [42, seed])
    q, _ = query_from(t, m, np.random.default_rng([43, seed]))
    with api.Engine(t) as e:
        for k in (1, 2, 3, 5, 10, 20):
            ci, cd, _ = e.cutoff(q, m, k, metric, 0, arg)
            oi, od, _ = oracle.cutoff(t, q, m, k, metric, 0, arg)
            assert list(ci) == list(oi) and bits_equal(cd, od), k
    scale, shift = 10.0 ** (seed - 4), (0.0, 833.0, 1e4)[seed % 3]
    t = walk_with_structure(6800, m, seed=[44, seed], nan_fraction=1e-3, flat_runs=4) * scale + shift
    q, _ = query_from(np.where(np.isfinite(t), t, shift), m, np.random.default_rng([45, seed]))
    oracle.set_normalization("raw")
    try:
        with api.Engine(t) as e:
            e.set_normalization("raw")
            for k in (1, 10, 60):
                ci, cd, _ = e.cutoff(q, m, k, metric, 8, arg * scale)
                oi, od, _ = oracle.cutoff(t, q, m, k, metric, 8, arg * scale)
                assert list(ci) == list(oi) and bits_equal(cd, od), k
    finally:
        oracle.set_normalization("zscore")


# The screen and the exact DP by the length of the list (screen_few, long_dp): lists
# on both sides of the lines, for the lane-per-candidate DP (w <= 20) and for MSM's
# widest bands (five to eight register chunks, m near 2w); cutoffs that the
# screen is used at and that it is not.  The lane DP is launched for the lists that
# may be long.
@pytest.mark.parametrize("metric,arg,m,w,n", [
    ("dtw", 0.0, 24, 2, 30_000), ("erp", 0.4, 24, 6, 30_000), ("msm", 0.5, 24, 6, 30_000), ("dtw", 0.0, 40, 20, 48_000),
    ("msm", 0.5, 24, 20, 48_000), ("dtw", 0.0, 24, 21, 12_000), ("msm", 0.5, 300, 140, 2600),
    ("msm", 0.5, 300, 165, 2600), ("msm", 0.5, 300, 200, 2600), ("msm", 0.5, 300, 240, 2600)])
def test_lists_behind_the_screen(api, oracle, metric, arg, m, w, n):  # noqa: F811
    import torch

    t = random_walk(n, [46, m, w])
    t[700] = np.nan
    q, _ = query_from(t, m, np.random.default_rng([47, m, w]))
    oi, od, oc = oracle.exact(t, q, m, 1e300, metric, w, arg)
    ranked = np.sort(od)
    d_t = torch.from_numpy(t).cuda()
    idx = torch.zeros(n, dtype=torch.int64, device="cuda")
    dist = torch.zeros(n, dtype=torch.float64, device="cuda")
    with api.Engine(t) as e:
        for cut in (ranked[20], ranked[len(ranked) // 2], ranked[-1], 1e6):
            keep = od <= cut
            e.exact(q, m, float(cut), metric, w, arg)
            e.set_profiling(True)
            gi, gd, gc = e.exact(q, m, float(cut), metric, w, arg)
            st = e.stage_times()
            e.set_profiling(False)
            assert list(gi) == list(oi[keep]) and gc["valid"] == oc["valid"], cut
            assert bits_equal(gd, od[keep]), cut
            si, sc = e.search(q, m, float(cut), metric, w, arg)
            yi, yc = oracle.search(t, q, m, float(cut), metric, w, arg)
            assert list(si) == list(yi) and sc["after_glb"] == yc["after_glb"], cut
            if w > 94:  # fsmeld_exact_noalloc takes no wider band
                continue
            c = api.exact_noalloc(d_t.data_ptr(), n, q, m, float(cut), metric, w, arg, idx.data_ptr(), dist.data_ptr(), n)
            assert c == keep.sum()
            assert np.array_equal(idx[:c].cpu().numpy(), oi[keep]) and bits_equal(dist[:c].cpu().numpy(), od[keep])
        if w <= 20:  # the last list holds every window
            assert st["k_dp"][1] == 1


# MSM's widest bands on long lists, by the kernel without interior steps in blocks of
# four warps (m large for the shared memory), on both sides of the lines for
# candidates that end early (m up to 3.5 w, 5.5 w); each chunk count from five on
@pytest.mark.parametrize("m,w", [(396, 159), (460, 165), (760, 200), (800, 240)])
def test_widest_bands_in_wide_blocks(api, oracle, m, w):  # noqa: F811
    n = m + 1900
    t = random_walk(n, [52, m, w])
    t[700] = np.nan
    q, _ = query_from(t, m, np.random.default_rng([53, m, w]))
    oi, od, oc = oracle.exact(t, q, m, 1e300, "msm", w, 0.5)
    ranked = np.sort(od)
    with api.Engine(t) as e:
        for cut in (0.5 * ranked[0], ranked[0], ranked[20], ranked[-1]):
            keep = od <= cut
            gi, gd, gc = e.exact(q, m, float(cut), "msm", w, 0.5)
            assert list(gi) == list(oi[keep]) and gc["valid"] == oc["valid"], cut
            assert bits_equal(gd, od[keep]), cut
            si, sc = e.search(q, m, float(cut), "msm", w, 0.5)
            yi, yc = oracle.search(t, q, m, float(cut), "msm", w, 0.5)
            assert list(si) == list(yi) and sc["after_glb"] == yc["after_glb"], cut


# Raw windows far off the query are dropped by the screen, four rows (ERP, MSM) or
# eight (DTW) into the band, and not handed on; ERP with a gap value further out than
# the points that the screen's bound covers
@pytest.mark.parametrize("metric,arg,w", [("dtw", 0.0, 12), ("erp", 0.4, 6), ("erp", 500.0, 6), ("msm", 0.0, 6), ("msm", 0.5, 6)])
def test_raw_windows_far_off(api, oracle, metric, arg, w):  # noqa: F811
    n, m = 300_000, 40
    rng = np.random.default_rng(54)
    t = np.where(np.arange(n) // 5000 % 2, 1.0, -1.0) * (300.0 + rng.normal(size=n))
    t[150_000:151_000] = random_walk(1000, 55)
    t[150_100] = 90.0  # one point out of range, and in a window that matches without it
    q = np.ascontiguousarray(t[150_300:150_340] + rng.normal(size=m) * 0.1)
    oracle.set_normalization("raw")
    try:
        oi, od, _ = oracle.exact(t[149_000:152_000], q, m, 1e300, metric, w, arg)
        with api.Engine(t) as e:
            e.set_normalization("raw")
            for cut in (np.sort(od)[0], np.sort(od)[30]):
                gi, gd, gc = e.exact(q, m, float(cut), metric, w, arg)
                keep = od <= cut
                assert list(gi) == list(oi[keep] + 149_000) and bits_equal(gd, od[keep]), cut
                rows = 8 if metric == "dtw" else 4
                if arg < 100:
                    assert gc["dp_cells"] < 1.5 * n * rows * (2 * w + 1), cut
    finally:
        oracle.set_normalization("zscore")


# Stage times: every launch has a record of its own (the matching table of EDR and
# LCSS counts with its DP), so no stage takes the time up to another's launch.
@pytest.mark.parametrize("metric", ["edr", "lcss", "dtw"])
def test_stage_records(api, metric):  # noqa: F811
    t = random_walk(20_000, 48)
    q, _ = query_from(t, 64, np.random.default_rng(49))
    spec = [dict(query=q, m=64, metric=metric, w=3, arg=0.25 if metric != "dtw" else 0.0, cutoff=0.5)] * 3
    with api.Engine(t) as e:
        e.set_concurrency(1)
        e.set_lb_form("fft")
        e.batch("search", spec)
        before = e.launches
        e.set_profiling(True)
        e.batch("search", spec)
        st = e.stage_times()
        e.set_profiling(False)
        assert sum(v[1] for v in st.values()) == e.launches - before
        assert st["k_bitdp"][1] == (0 if metric == "dtw" else 6)


# LB_IP by the changes of the masks, against the products in extended precision:
# off by the fixed-point rounding of each penalty (m/2 units of 2^-60 m h_max a
# side), the two conversions and, squared again here, the root.  Noise (a change at
# nearly every position), walks, raw series of large values and with spikes that
# become thresholds.
@pytest.mark.parametrize("kind", ["walk", "noise", "raw", "spikes"])
@pytest.mark.parametrize("m,w", [(16, 0), (100, 0), (200, 1), (1000, 9), (512, 26)])
@pytest.mark.parametrize("metric,arg", [("dtw", 0.0), ("erp", 0.4), ("msm", 0.5)])
def test_mask_changes_in_extended_precision(api, oracle, metric, arg, m, w, kind):  # noqa: F811
    mk = 1
    while mk < 8 * m:
        mk *= 2
    kml = mk - m + 1
    t = np.random.default_rng([50, m]).normal(size=2 * kml + m) if kind == "noise" else random_walk(2 * kml + m, [50, m])
    raw = kind in ("raw", "spikes")
    q, _ = query_from(t, m, np.random.default_rng([51, m]))
    if kind == "raw":
        t, q = t * 1e4 + 1e5, q * 1e4 + 1e5
    if kind == "spikes":
        t[[kml // 3, kml + kml // 2]] += [1e12, -1e12]
    x = np.asarray(q) if raw else oracle.normalize_query(q)
    with api.Engine(t) as e:
        e.set_normalization("raw" if raw else "zscore")
        z = e.inspect(q, m, metric, w, arg, 5).reshape(-1, kml)
        thr = e.inspect(q, m, metric, w, arg, 4).reshape(-1, 2)
        un = e.inspect(q, m, metric, w, arg, 2).reshape(-1, mk)
        ln = e.inspect(q, m, metric, w, arg, 3).reshape(-1, mk)
    for s in range(2):
        tl, tu = thr[s]
        h = [oracle.q_to_h(u, metric, x, thr[s, u], arg).astype(np.longdouble) for u in (0, 1)]
        g = [ln[s] >= tl, un[s] <= tu]
        ref = np.zeros(kml, dtype=np.longdouble)
        for u in (0, 1):
            for k in range(m):
                ref += h[u][k] * g[u][k:k + kml]
        far = [max(0.0, tl - x.min()), max(0.0, x.max() - tu)]
        hmax = [min(f, arg) if metric == "msm" else f * f for f in far]
        if metric == "erp":
            hmax = [min(v, max((x.min() - arg) ** 2, (x.max() - arg) ** 2)) for v in hmax]
        tol = sum(0.5 * m * 2.0 ** -60 * m * v for v in hmax) + 2.0 ** -50 * ref
        got = z[s].astype(np.longdouble)
        ok = ~np.isnan(got)
        err = np.abs((got if metric == "msm" else got * got) - ref)
        assert ok.any() and np.all(err[ok] <= tol[ok]), (s, float((err[ok] / tol[ok]).max()))


# The bit vectors with outliers among the query's points: nearly all ends of the
# matching intervals in one bucket of the lookup (bisected there), windows with
# and without the outlier, points on and beside the ends.  On its time: 30 times
# that of the same query without the outlier when the bucket was stepped through.
@pytest.mark.parametrize("spike", [50.0, -1e3, 1e9])
@pytest.mark.parametrize("metric,arg", [("edr", 0.25), ("lcss", 0.25), ("edr", 0.0), ("lcss", 2.0)])
def test_bit_vectors_with_outliers(api, oracle, metric, arg, spike):  # noqa: F811
    m, w = 700, 9
    t = np.round(random_walk(3500, 55), 2)
    t[900] += spike
    q = t[800:800 + m].copy()
    q[::7] += 0.25
    oracle.set_normalization("raw")
    try:
        with api.Engine(t) as e:
            e.set_normalization("raw")
            for cut in (1e300, 0.6 if metric == "lcss" else 300.0):
                gi, gd, gc = e.exact(q, m, cut, metric, w, arg)
                oi, od, oc = oracle.exact(t, q, m, cut, metric, w, arg)
                assert list(gi) == list(oi) and bits_equal(gd, od) and gc["valid"] == oc["valid"]
            ci, cd, _ = e.cutoff(q, m, 20, metric, w, arg)
            oi, od, _ = oracle.cutoff(t, q, m, 20, metric, w, arg)
            assert list(ci) == list(oi) and bits_equal(cd, od)

            def scan(query):
                times = []
                for _ in range(5):
                    e.exact(query, m, 1e300, metric, w, arg)
                    times.append(e.last_call_ms)
                return min(times)

            plain = q.copy()
            plain[100] = plain[99]
            assert scan(q) < 4.0 * scan(plain)
    finally:
        oracle.set_normalization("zscore")


# Raw series on which FP32 proves nothing (values far from zero against their
# differences) are not screened, those of tiny values are: either way the scan does
# less than the cells of one full band a window.
@pytest.mark.parametrize("scale,shift", [(1e-9, 5.0), (1e-9, 0.0), (1.0, 1e7)])
@pytest.mark.parametrize("metric,arg,w", [("dtw", 0.0, 25), ("erp", 0.0, 25), ("msm", 0.1, 25), ("dtw", 0.0, 5)])
def test_raw_series_beyond_fp32(api, oracle, metric, arg, w, scale, shift):  # noqa: F811
    n, m = 30_000, 120
    t = random_walk(n, 56) * scale + shift
    q = t[700:700 + m] + np.random.default_rng(57).normal(0.0, 0.1, m) * scale
    oracle.set_normalization("raw")
    try:
        with api.Engine(t) as e:
            e.set_normalization("raw")
            _, d, _ = e.cutoff(q, m, 20, metric, w, arg * scale)
            gi, gd, c = e.exact(q, m, float(d[-1]), metric, w, arg * scale)
            oi, od, _ = oracle.exact(t, q, m, float(d[-1]), metric, w, arg * scale)
            assert list(gi) == list(oi) and bits_equal(gd, od)
            _, _, c = e.exact(q, m, 0.0, metric, w, arg * scale)
            assert c["dp_cells"] < (n - m) * m * (2 * w + 1)
    finally:
        oracle.set_normalization("zscore")



# Top-k past the wavefront's and the bit vectors' bands: the seeds' distances and the
# survivors', no refining windows between (a launch more of one lane a window)
@pytest.mark.parametrize("metric,arg", [("dtw", 0.0), ("msm", 0.5), ("lcss", 0.25)])
def test_widest_bands_are_not_refined(api, oracle, metric, arg):  # noqa: F811
    m, w = 280, 260
    t = random_walk(1500, 58)
    q, _ = query_from(t, m, np.random.default_rng(59))
    with api.Engine(t) as e:
        e.set_profiling(True)
        ci, cd, _ = e.cutoff(q, m, 5, metric, w, arg)
        st = e.stage_times()
        e.set_profiling(False)
    oi, od, _ = oracle.cutoff(t, q, m, 5, metric, w, arg)
    assert list(ci) == list(oi) and bits_equal(cd, od)
    assert st["k_dp"][1] == 2


# m = 2: GLB is its boundary alone, and the reference abandons at inner points only;
# cutoffs at the distances themselves, where the square's rounding decides
@pytest.mark.parametrize("metric,arg", [("dtw", 0.0), ("erp", 0.4), ("msm", 0.5), ("edr", 0.25), ("lcss", 0.25)])
@pytest.mark.parametrize("seed", range(4))
def test_two_points(api, oracle, metric, arg, seed):  # noqa: F811
    t = np.round(random_walk(400, [60, seed])) if seed < 2 else random_walk(400, [60, seed])
    q = np.array([0.3, -1.1]) if seed % 2 else t[50:52] + np.array([0.01, -0.02])
    raw = seed >= 2
    oracle.set_normalization("raw" if raw else "zscore")
    try:
        with api.Engine(t) as e:
            e.set_normalization("raw" if raw else "zscore")
            _, od, _ = oracle.exact(t, q, 2, 1e300, metric, 0, arg)
            for cut in np.unique(od)[:12]:
                si, sc = e.search(q, 2, float(cut), metric, 0, arg)
                oi, oc = oracle.search(t, q, 2, float(cut), metric, 0, arg)
                assert list(si) == list(oi) and sc["after_glb"] == oc["after_glb"], cut
    finally:
        oracle.set_normalization("zscore")
