"""Requests close to the server's memory budget: what was admitted when the host built every field grid is
admitted, with the plain result."""
import numpy as np
import pytest

from optixsoltracedemos_gb300 import native, scenes

pytestmark = pytest.mark.gpu


# heliostats, own poses, spread of the field, the block of such a request with a host-built field grid of
# 4-byte cell starts and no reach raster (100 x 100 bins)
@pytest.mark.parametrize("heliostats,own,spread,block", [
    (20, True, 1.0, 65_536), (100, True, 1.0, 140_544), (1000, True, 1.0, 983_808), (1000, True, 4.0, 1_604_864),
    (10_000, True, 1.0, 9_009_664), (20, False, 1.0, 58_880), (1000, False, 1.0, 705_792)])
def test_request_close_to_the_budget(gpu, heliostats, own, spread, block):
    elements = scenes.large_field(n_heliostats=heliostats, sun=scenes.sun_vector(45.0, 0.0), num_rays=1).elements
    elements["origin"][:-1, :2] *= spread
    sun = scenes.sun_vector(50.0, 10.0)
    poses = scenes.reaim(elements, sun) if own else None
    rays = 100_000
    maps = []
    for budget in (256 << 20, block):
        srv = native.Server(0, memory_budget=budget, max_active=4)
        sid = srv.add_scene(elements)
        rid = srv.submit(sid, sun, scenes.SUN_PILLBOX, 4.65e-3, rays, seed=3, instance=2, poses=poses)
        maps.append(srv.wait(rid, timeout=60.0)[0])
        assert srv.stats()["peak_arena_bytes"] <= budget
        srv.close()
    t = native.Tracer(0, rays)
    t.set_elements(elements if poses is None else poses)
    t.set_sun_vector(sun)
    t.set_sun_shape(scenes.SUN_PILLBOX, 4.65e-3)
    t.set_seed(3, 2)
    t.initialize()
    t.run()
    want, _ = t.flux_map(100, 100)
    t.close()
    assert want.any() or spread > 1.0
    for m in maps:
        np.testing.assert_array_equal(m, want)


def test_exact_items_fit_where_the_bound_does_not(gpu):
    """Between the two sizes the request keeps its grid: the exact items, counted on the host, hold what the
    device registers."""
    elements = scenes.large_field(n_heliostats=1000, sun=scenes.sun_vector(45.0, 0.0), num_rays=1).elements
    sun = scenes.sun_vector(50.0, 10.0)
    poses = scenes.reaim(elements, sun)

    def served(budget):
        srv = native.Server(0, memory_budget=budget, max_active=4)
        sid = srv.add_scene(elements)
        rid = srv.submit(sid, sun, scenes.SUN_PILLBOX, 4.65e-3, 200_000, seed=3, poses=poses)
        counts = srv.wait(rid, timeout=60.0)[0]
        peak = int(srv.stats()["peak_arena_bytes"])
        srv.close()
        return counts, peak

    counts, full = served(64 << 20)
    tight_counts, tight = served(full - 256)
    assert 983_808 < tight < full
    np.testing.assert_array_equal(tight_counts, counts)
    assert counts.any()
