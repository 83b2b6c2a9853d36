"""Batch instances around the block sizes of the coherent ray order (55,296 rays and 331,776), and scene
set-up around the sizes at which it changes form: flux maps equal the oracle's."""
import numpy as np
import pytest

from optixsoltracedemos_gb300 import native, scenes

pytestmark = pytest.mark.gpu

B3, B2 = 55_296, 331_776


def _field(n, slope=0.0, spread=1.0):
    sun = scenes.sun_vector(50.0, -20.0)
    e = scenes.large_field(n_heliostats=n, sun=sun, num_rays=1).elements
    e["origin"][:-1, :2] *= spread
    e["origin"][:, 2] += slope * e["origin"][:, 1]
    e["aim_point"][-1] = e["origin"][-1] + [0.0, -1.0, 0.0]
    return scenes.reaim(e, sun), sun


def _check(oracle32, elements, sun, counts, block):
    b = native.Batch(0)
    sid = b.add_scene(elements)
    for i, rays in enumerate(counts):
        b.add_instance(sid, sun, scenes.SUN_PILLBOX, 4.65e-3, rays, seed=7, instance=i, poses=elements)
    b.set_tuning(block, 0, 16)
    b.run()
    target = native.flux_target(elements[-1])
    for i, rays in enumerate(counts):
        oh, _ = oracle32.trace(elements, sun, scenes.SUN_PILLBOX, 4.65e-3, count=rays, seed=7, instance=i)
        want, _ = oracle32.flux_counts(oh.astype(np.float32), target)
        np.testing.assert_array_equal(b.counts(i), want)
        assert want.any()
    b.close()


@pytest.mark.parametrize("slope", [0.0, 0.6], ids=["grid", "bvh"])
@pytest.mark.parametrize("block", [128, 256])
def test_instances_around_the_order_blocks(gpu, oracle32, slope, block):
    elements, sun = _field(20, slope)
    _check(oracle32, elements, sun, [B3 - 1, B3, B3 + 1, 2 * B3 + 257, B2 - 1, B2 + B3 + 37], block)


# 1,023 and 1,024 elements, and a field so wide that its grid has 10^5 cells
@pytest.mark.parametrize("heliostats,spread,rays", [(1022, 1.0, 20_000), (1023, 1.0, 20_000), (30, 24.0, 1_000_000)])
def test_instances_around_the_set_up_forms(gpu, oracle32, heliostats, spread, rays):
    elements, sun = _field(heliostats, spread=spread)
    _check(oracle32, elements, sun, [rays, rays + 5], 256)
