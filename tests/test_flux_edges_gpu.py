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


@pytest.mark.parametrize("tuning", [(128, 0, 1), (256, 0, 1 << 30)])
@pytest.mark.parametrize("name", ["three_heliostats", "single_parabolic"])
def test_batch_record_counters(gpu, oracle32, name, tuning):
    """Record counters of batch instances, kept per grab of tiles: grabs of one tile and as large as they
    get, instances smaller than a CTA among them; equal to the oracle's counts."""
    rays = [1, 100, 200_003]
    sc = getattr(scenes, name)(num_rays=1)
    b = native.Batch(0, 100, 100)
    sid = b.add_scene(sc.elements)
    for k, n in enumerate(rays):
        b.add_instance(sid, sc.sun_dir, sc.sun_shape, sc.sun_param, n, seed=5, instance=k)
    b.set_tuning(*tuning)
    b.run()
    target = native.flux_target(sc.elements[-1])
    for k, n in enumerate(rays):
        oh, _ = oracle32.trace(sc.elements, sc.sun_dir, sc.sun_shape, sc.sun_param, 0, n, seed=5, instance=k)
        counts, _ = oracle32.flux_counts(oh.astype(np.float32), target)
        np.testing.assert_array_equal(b.counts(k), counts)
        want = [n, (oh[..., 0] == 1.0).sum(), (oh[..., 0] == 2.0).sum(), counts.sum()]
        assert [int(v) for v in b.stats(k)] == [int(v) for v in want]
    b.close()


@pytest.mark.parametrize("bins", [100, 700])
def test_map_without_pinned_memory(gpu, bins):
    """Where no pinned memory is to be had the map is the same."""
    sc = scenes.large_field(n_heliostats=50, sun=scenes.sun_vector(45.0, 10.0))
    maps = []
    for fail in (False, True):
        t = native.tracer_for(sc, seed=1, num_rays=200_000)
        t.run()
        t.flux_map(2, 2)  # the map on the device and its pinned copy are to grow
        for k in range(3):
            if fail:
                native.debug_fail_allocation(1 if k == 0 else 0)  # the second allocation of the first call
            try:
                maps.append(t.flux_map(bins, bins)[0])
            finally:
                native.debug_fail_allocation(-1)
        t.close()
    assert maps[0].any()
    for m in maps[1:]:
        np.testing.assert_array_equal(m, maps[0])
