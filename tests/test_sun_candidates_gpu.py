"""Sun-ray candidates of scenes above 8 elements (reach raster, then candidate rectangles around the
crossing of a reference plane) at their edges: every record and element id equals the oracle's
brute-force closest hit bit for bit."""
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
}


@pytest.mark.parametrize("name", list(CASES))
def test_sun_candidates_bit_exact(gpu, oracle32, name):
    sc = CASES[name]()
    n = 30000
    oh, oi = oracle32.trace(sc.elements, sc.sun_dir, sc.sun_shape, sc.sun_param, count=n, seed=13, instance=1)
    t = native.tracer_for(sc, seed=13, instance=1, num_rays=n)
    t.run()
    hits, ids = t.copy_hits()
    t.close()
    np.testing.assert_array_equal(ids, oi)
    np.testing.assert_array_equal(hits, oh.astype(np.float32))
    assert (oh[:, 1:, 0] != 0).any()
