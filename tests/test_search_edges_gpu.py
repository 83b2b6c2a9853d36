"""Closest-hit search of scenes above 8 elements at its edges: sun-ray candidates (reach raster, then
candidate rectangles around the crossing of a reference plane) and reflections (which pass over the
flat mirror they leave).  Every record and element id equals the oracle's brute-force closest hit bit
for bit, through the field grid and the BVH."""
import numpy as np
import pytest

from optixsoltracedemos_gb300 import native, scenes

pytestmark = pytest.mark.gpu


def _stack():
    """12 mirrors above each other: no level layer, the reference plane lies across the sun."""
    e = scenes.make_elements(13)
    e["origin"][:12] = [[0.0, 0.0, 10.0 * k] for k in range(12)]
    e["aim_point"][:12] = [[0.0, 1.0, 10.0 * k + 1.0] for k in range(12)]
    e["width"][:12] = e["height"][:12] = 5.0
    e["origin"][12], e["aim_point"][12] = [0.0, 50.0, 50.0], [0.0, 0.0, 50.0]
    e["width"][12] = e["height"][12] = 10.0
    return scenes.Scene("stack", e, np.array([0.0, 1.0, 0.2]), scenes.SUN_PILLBOX, 4.65e-3, 1)


def _field(n, el, az=30.0, offset=0.0, slope=0.0, **kw):
    sun = scenes.sun_vector(el, az)
    sc = scenes.large_field(n_heliostats=n, sun=sun, **kw)
    sc.elements["origin"] += [offset, -offset, 0.0]
    sc.elements["origin"][:, 2] += slope * sc.elements["origin"][:, 1]
    sc.elements["aim_point"][-1] = sc.elements["origin"][-1] + [0.0, -1.0, 0.0]
    sc.elements = scenes.reaim(sc.elements, sun)
    return sc


def _facing(n, el, normal, step, specularity=0.0):
    """A row of n large mirrors that all face `normal`: chosen incidences, up to grazing."""
    e = scenes.make_elements(n + 1)
    e["origin"][:n] = [[step * k, 0.0, 0.0] for k in range(n)]
    e["origin"][n] = [0.5 * n * step, 60.0, 40.0]
    e["aim_point"][:n] = e["origin"][:n] + np.asarray(normal)
    e["aim_point"][n] = e["origin"][n] - [0.0, 1.0, 0.3]
    e["width"], e["height"] = 8.0, 8.0
    e["width"][n] = e["height"][n] = 60.0
    e["slope_error"][:n], e["specularity_error"][:n] = 2e-2, specularity
    return scenes.Scene("facing", e, scenes.sun_vector(el, 0.0), scenes.SUN_PILLBOX, 4.65e-3, 1)


def _walls():
    """Two walls of five mirrors facing each other: paths of several reflections."""
    e = scenes.make_elements(11)
    for k in range(5):
        e["origin"][k], e["aim_point"][k] = [-2.0, 4.0 * k, 0.0], [1.0, 4.0 * k, 0.0]
        e["origin"][5 + k], e["aim_point"][5 + k] = [2.0, 4.0 * k, 0.0], [-1.0, 4.0 * k, 0.0]
    e["width"], e["height"], e["slope_error"] = 20.0, 4.0, 1e-3
    e["origin"][10], e["aim_point"][10] = [0.0, 8.0, -10.5], [0.0, 8.0, 0.0]
    return scenes.Scene("walls", e, np.array([0.8, 0.1, 1.0]), scenes.SUN_PILLBOX, 4.65e-3, 1)


def _mixed_sizes(ratio):
    """Mirrors of two sizes: the device builds the field grid up to boxes 11.2 times the smallest."""
    sc = _field(150, 35.0)
    sc.elements["width"][:150:3] = sc.elements["height"][:150:3] = 10.0 / ratio
    return sc


CASES = {
    "nine_elements": lambda: _field(8, 35.0),
    # the sun frame is one block below 1,024 elements, a cluster from there
    "elements_1023": lambda: _field(1022, 50.0),
    "elements_1024": lambda: _field(1023, 50.0),
    # level plane above about 1.2 degrees of sun elevation, across the sun below
    "sun_1_deg": lambda: _field(120, 1.0),
    "sun_2_deg": lambda: _field(120, 2.0),
    "stack": _stack,
    "slope": lambda: _field(200, 40.0, slope=0.6),
    # coordinates far from the origin: the margins against rounding
    "offset_20_km": lambda: _field(200, 25.0, offset=2e4),
    # the field grid: device-built, and on the host past the limits of sizes and of coordinates
    "mixed_sizes_4": lambda: _mixed_sizes(4.0),
    "mixed_sizes_40": lambda: _mixed_sizes(40.0),
    "offset_90_km": lambda: _field(200, 60.0, offset=9e4),
    # incidences around the limit of the own-mirror rule and beyond it, mirrors facing each other
    "incidence_65_deg": lambda: _facing(12, 25.0, [0.0, 0.0, 1.0], 9.0),
    "incidence_85_deg": lambda: _facing(12, 5.0, [0.0, 0.0, 1.0], 9.0, specularity=5e-2),
    "walls": _walls,
}


@pytest.mark.parametrize("accel", [native.ACCEL_AUTO, native.ACCEL_BVH], ids=["auto", "bvh"])
@pytest.mark.parametrize("name", list(CASES))
def test_search_edges_bit_exact(gpu, oracle32, name, accel):
    sc = CASES[name]()
    n = 30000
    oh, oi = oracle32.trace(sc.elements, sc.sun_dir, sc.sun_shape, sc.sun_param, count=n, seed=13, instance=1)
    t = native.tracer_for(sc, seed=13, instance=1, num_rays=n, accel=accel)
    t.run()
    hits, ids = t.copy_hits()
    t.close()
    np.testing.assert_array_equal(ids, oi)
    np.testing.assert_array_equal(hits, oh.astype(np.float32))
    assert (oh[:, 1:, 0] != 0).any()


def test_update_between_grid_and_bvh(gpu, oracle32):
    """update() of a planar field to steep ground and back: the BVH is built when it is first needed."""
    flat, steep = _field(300, 40.0), _field(300, 40.0, slope=0.6)
    n = 20000
    t = native.tracer_for(flat, seed=5, num_rays=n)
    for sc, accel in ((flat, native.ACCEL_GRID), (steep, native.ACCEL_BVH), (flat, native.ACCEL_GRID),
                      (steep, native.ACCEL_BVH)):
        t.set_elements(sc.elements)
        t.update()
        assert t.accel() == accel
        t.run()
        hits, ids = t.copy_hits()
        oh, oi = oracle32.trace(sc.elements, sc.sun_dir, sc.sun_shape, sc.sun_param, count=n, seed=5)
        np.testing.assert_array_equal(ids, oi)
        np.testing.assert_array_equal(hits, oh.astype(np.float32))
    # an update that is refused leaves the scene as it was
    t.set_accel(native.ACCEL_GRID)
    t.set_elements(flat.elements)
    t.initialize()
    bad = flat.elements.copy()
    bad["width"][7] = -1.0
    for refused in (bad, steep.elements):
        t.set_elements(refused)
        with pytest.raises(native.CspError):
            t.update()
    t.run()
    hits, ids = t.copy_hits()
    oh, oi = oracle32.trace(flat.elements, flat.sun_dir, flat.sun_shape, flat.sun_param, count=n, seed=5)
    np.testing.assert_array_equal(ids, oi)
    np.testing.assert_array_equal(hits, oh.astype(np.float32))
    t.close()
