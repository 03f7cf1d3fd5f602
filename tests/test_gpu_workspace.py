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
