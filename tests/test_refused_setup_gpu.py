"""initialize() and update() that are refused or fail: the scene that the device holds stays as it was and
traceable, whatever the element count of the refused one."""
import numpy as np
import pytest

from optixsoltracedemos_gb300 import native, scenes

pytestmark = pytest.mark.gpu

RAYS = 20_000


def _field(heliostats, slope=0.0):
    sc = scenes.large_field(n_heliostats=heliostats, sun=scenes.sun_vector(45.0, 20.0))
    if slope:
        sc.elements["origin"][:, 2] += slope * sc.elements["origin"][:, 1]
        sc.elements["aim_point"][:, 2] += slope * sc.elements["origin"][:, 1]
    return sc


def _expect(t, sc, oracle32, rays=RAYS):
    t.run()
    hits, ids = t.copy_hits()
    oh, oi = oracle32.trace(sc.elements, sc.sun_dir, sc.sun_shape, sc.sun_param, count=rays, seed=5)
    np.testing.assert_array_equal(ids, oi)
    np.testing.assert_array_equal(hits, oh.astype(np.float32))


# element counts (heliostats and receiver) held and refused: list, grid, both ways, larger buffers, host
# threads; refused for a bad element or (above 8 elements) for poses that ACCEL_GRID cannot take
COUNTS = [(20, 5), (5, 3), (3, 4), (5, 20), (20, 300), (300, 9), (300, 5000)]


@pytest.mark.parametrize("held,refused,why", [(*c, "element") for c in COUNTS] +
                         [(*c, "plan") for c in COUNTS if c[1] > 8])
def test_refused_initialize_keeps_the_scene(gpu, oracle32, held, refused, why):
    sc = _field(held - 1)
    t = native.tracer_for(sc, seed=5, num_rays=RAYS, accel=native.ACCEL_GRID)
    new = _field(refused - 1, slope=0.6 if why == "plan" else 0.0).elements
    if why == "element":
        new["width"][refused - 2] = -1.0
    t.set_elements(new)
    with pytest.raises(native.CspError) as e:
        t.initialize()
    assert e.value.status == -4, str(e.value)  # CSP_ERR_BAD_SCENE
    _expect(t, sc, oracle32)
    with pytest.raises(native.CspError):  # not the count of the scene held
        t.update()
    _expect(t, sc, oracle32)
    t.set_elements(sc.elements)
    t.update()
    _expect(t, sc, oracle32)
    t.close()


@pytest.mark.parametrize("heliostats", [4, 300])
def test_update_without_memory_for_the_records(gpu, oracle32, heliostats):
    """More rays than memory for their records: update() fails, and fewer rays trace its scene."""
    sc = _field(heliostats)
    t = native.tracer_for(sc, seed=5, num_rays=RAYS)
    moved = scenes.reaim(sc.elements, scenes.sun_vector(50.0, -10.0))
    sc.elements, sc.sun_dir = moved, scenes.sun_vector(50.0, -10.0)
    t.set_elements(moved)
    t.set_sun_vector(sc.sun_dir)
    t.set_num_rays(2 * RAYS)
    native.debug_fail_allocation(0)
    try:
        with pytest.raises(native.CspError) as e:
            t.update()
        assert e.value.status == -3
    finally:
        native.debug_fail_allocation(-1)
    t.set_num_rays(RAYS)
    _expect(t, sc, oracle32)
    t.close()


@pytest.mark.parametrize("accel", [native.ACCEL_GRID, native.ACCEL_BVH])
def test_update_that_fails_can_be_repeated(gpu, oracle32, accel):
    """A re-initialize() whose k-th allocation fails traces nothing; update() alone completes it."""
    small, sc = _field(20), _field(300)
    for k in range(16):
        t = native.tracer_for(small, seed=5, num_rays=RAYS, accel=accel)
        t.run()
        t.set_elements(sc.elements)
        native.debug_fail_allocation(k)
        try:
            t.initialize()
            failed = False
        except native.CspError as e:
            assert e.status == -3
            failed = True
        finally:
            native.debug_fail_allocation(-1)
        if not failed:
            assert k >= 2
            break
        assert t.copy_hits()[0].any()  # the last run's
        if k < 2:  # the element records' buffers: before the new scene is accepted
            _expect(t, small, oracle32)
            t.initialize()
        else:
            with pytest.raises(native.CspError) as e:
                t.run()
            assert e.value.status == -6
            t.update()
        _expect(t, sc, oracle32)
        t.close()
