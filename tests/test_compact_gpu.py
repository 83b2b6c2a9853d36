"""Compact records at the edges of their chunks (a quarter of the run, 131,072 to 1,048,576 rays) and through
the one-piece path (a capacity that some run could exceed): points, counts and records are the dense
buffer's, and a capacity that is too small copies nothing."""
import numpy as np
import pytest

from optixsoltracedemos_gb300 import native, scenes

pytestmark = pytest.mark.gpu


def _dense(t):
    hits, _ = t.copy_hits()
    used = hits[:, 1:, 0] != 0
    return hits[:, 0, 1:], used.sum(1).astype(np.uint8), hits[:, 1:][used]


@pytest.mark.parametrize("n", [1, 255, 1 << 17, (1 << 17) + 1, 3 * (1 << 17), 5 * (1 << 18) - 77, (1 << 21) + 12345, 9 * (1 << 19) + 1])
def test_compact_chunks(gpu, n):
    sc = scenes.corridor(slope_error=1e-3)  # up to four records a ray
    t = native.tracer_for(sc, seed=4, num_rays=n, record_ids=False)
    for capacity in (4 * n, 4 * n - 1):  # chunks, one piece
        points, counts, records = t.run_to_host_compact(records=np.empty((capacity, 4), np.float32))
        p, c, r = _dense(t)
        np.testing.assert_array_equal(points, p)
        np.testing.assert_array_equal(counts, c)
        np.testing.assert_array_equal(records, r)
    if len(r):
        sentinel = np.full((n, 3), -7.0, np.float32)
        with pytest.raises(native.CspError):
            t.run_to_host_compact(points=sentinel, records=np.empty((len(r) - 1, 4), np.float32))
        assert (sentinel == -7.0).all()
    t.close()


@pytest.mark.parametrize("n", [655_359, 655_360, 983_039, 983_041, 1_310_720, (1 << 22) + 257])
def test_compact_parts(gpu, n):
    """Runs around the sizes at which they get another part, and past four parts of 2^20 rays."""
    sc = scenes.corridor(slope_error=1e-3)
    t = native.tracer_for(sc, seed=6, num_rays=n, record_ids=False)
    points, counts, records = t.run_to_host_compact(records=np.empty((4 * n, 4), np.float32))
    p, c, r = _dense(t)
    np.testing.assert_array_equal(points, p)
    np.testing.assert_array_equal(counts, c)
    np.testing.assert_array_equal(records, r)
    t.close()
