"""Calls at workspace limits: what a call cannot do without is all that it asks
for (needs a B200)."""
import numpy as np
import pytest

from fsmeld_b200.synth import query_from, random_walk
from tests.test_gpu_parity import _geom, api, bits_equal  # noqa: F401

pytestmark = pytest.mark.gpu


# The exact scan: statistics, results (index and distance per window) and small
# buffers.  The FP32 screen's list is used where there is room, not asked for.
@pytest.mark.parametrize("metric,arg", [("dtw", 0.0), ("erp", 0.4), ("msm", 0.5), ("edr", 0.25), ("lcss", 0.25)])
def test_exact_asks_for_no_screen_list(api, metric, arg):  # noqa: F811
    n, m, w = 200_000, 100, 5
    t = random_walk(n, 51)
    q, _ = query_from(t, m, np.random.default_rng(52))
    _, kml, forsize, tail = _geom(m, n)
    need = 16 * (forsize + (tail > 0)) * kml + 16 * (n - m + 1)
    with api.Engine(t) as e:
        i, d, _ = e.cutoff(q, m, 30, metric, w, arg)
        want = e.exact(q, m, float(d[-1]), metric, w, arg)
    with api.Engine(t) as e:
        e.set_workspace_limit(need * 9 // 8 + (256 << 10))
        for _ in range(2):
            gi, gd, c = e.exact(q, m, float(d[-1]), metric, w, arg)
            assert np.array_equal(gi, want[0]) and bits_equal(gd, want[1]) and c["valid"] == want[2]["valid"]
        e.set_workspace_limit(0)
        gi, gd, _ = e.exact(q, m, float(d[-1]), metric, w, arg)
        assert np.array_equal(gi, want[0]) and bits_equal(gd, want[1])


# GLB's FP32 rows (2^18 points and more) under a workspace limit: a limit without room
# for them beside the query's lists costs the rows, not a second run; one with room
# has them.  Single searches and top-k, a group of one length, mixed lengths.
@pytest.mark.parametrize("room", [False, True])
@pytest.mark.parametrize("mode", ["search", "cutoff"])
@pytest.mark.parametrize("lengths", [[100], [100, 100, 100], [100, 70]])
def test_rows_beside_the_lists(api, mode, lengths, room):  # noqa: F811
    n, w = 300_000, 5
    t = random_walk(n, 53)
    qs, shared, own, rows = [], 0, 0, 0
    for i, m in enumerate(lengths):
        q, _ = query_from(t, m, np.random.default_rng([54, i]))
        qs.append(dict(query=q, m=m, metric="dtw", w=w, arg=0.0, k=20, cutoff=0.1 * m ** 0.5))
        mk, kml, forsize, tail = _geom(m, n)
        S = forsize + (tail > 0)
        env = 16 * S * kml + 16 * S * mk + 16 * n
        row = 12 * S * mk + 16 * S
        lists = 64 * n + (8 * S * kml if mode == "cutoff" else 0) + 80 * S
        apart = len(set(lengths)) > 1  # a worker each, with its own envelopes
        shared, rows = (shared + env, rows + row) if apart else (env, row)
        own += lists
    need = (shared + own) * 9 // 8 + len(qs) * (9 << 18) + (1 << 20)
    want = rows * 9 // 8
    with api.Engine(t) as e:
        ref = e.batch(mode, qs)
    with api.Engine(t) as e:
        e.set_workspace_limit(need + (want * 5 // 4 if room else want // 3))
        e.set_profiling(True)
        got = e.batch(mode, qs)
        st = e.stage_times()
        e.set_profiling(False)
    for g, r in zip(got, ref):
        assert g["status"] == 0
        assert np.array_equal(g["idx"], r["idx"]) and bits_equal(g["dist"], r["dist"])
    assert st["k_threshold"][1] == len(qs)  # no query ran twice
    envelopes = len(set(lengths))
    assert st["k_fwd_env"][1] == envelopes * (2 if room else 1)
