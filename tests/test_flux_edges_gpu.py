"""csp_flux_map at the edges of its record pass (spans of 1,024 records, batches of 32 receiver hits per
warp): counts equal the oracle's binning of the same records, staged and not."""
import numpy as np
import pytest

from optixsoltracedemos_gb300 import native, scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 204, 205, 7001])
@pytest.mark.parametrize("name", ["three_heliostats", "single_parabolic"])
def test_flux_map_edges(gpu, oracle32, name, n):
    sc = getattr(scenes, name)()
    sc.elements["width"][-1] *= 4  # a larger receiver: direct sun on it, more hits
    t = native.tracer_for(sc, seed=3, num_rays=n)
    t.run()
    hits, _ = t.copy_hits()
    target = native.flux_target(sc.elements[-1], 37, 23)
    for staged in (False, True):
        recs = hits.copy()
        if staged:
            recs[recs[:, 1, 0] == 2.0, 1] = 0.0
        counts, _ = t.flux_map(37, 23, staged=staged)
        np.testing.assert_array_equal(counts, oracle32.flux_counts(recs, target, 37, 23)[0])
    t.close()
