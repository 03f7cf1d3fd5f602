"""Kernels at the edges of their tiles, against the oracle (needs a B200):
lengths around the tile widths, macro segments clipped to the target, odd
segment counts, non-finite points on tile borders.  Window statistics,
envelopes, thresholds and distances are compared bit for bit."""
import numpy as np
import pytest

from fsmeld_b200.synth import query_from, random_walk
from tests.test_gpu_parity import _segments, api, bits_equal  # noqa: F401

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
