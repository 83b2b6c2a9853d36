"""The host work of a batch is spread over the batch's threads whether its instances have poses of their own
or share the scene's."""
import os

import numpy as np
import pytest

from optixsoltracedemos_gb300 import native, scenes

pytestmark = pytest.mark.gpu


def _threads():
    return len(os.listdir("/proc/self/task"))


@pytest.mark.parametrize("own", [False, True])
def test_large_runs_use_host_threads(gpu, own):
    field = scenes.large_field(n_heliostats=2000, num_rays=1).elements
    suns = [scenes.sun_vector(30.0 + 3 * i, -40.0 + 5 * i) for i in range(16)]

    def run(which):
        b = native.Batch(0)
        sid = b.add_scene(field)
        for i in which:
            b.add_instance(sid, suns[i], scenes.SUN_PILLBOX, 4.65e-3, 30_001 + i, seed=i, instance=i,
                           poses=scenes.reaim(field, suns[i]) if own else None)
        b.set_tuning(256, 0, 16)
        before = _threads()
        b.run()
        return b, [b.counts(k) for k in range(len(which))], _threads() - before

    alone = []
    for i in (0, 7, 15):  # one instance: nothing to spread; also brings up the driver's own threads
        b, counts, _ = run([i])
        alone.append(counts[0])
        b.close()
    b, counts, started = run(range(16))
    assert os.cpu_count() == 1 or started >= 1
    for want, i in zip(alone, (0, 7, 15)):
        np.testing.assert_array_equal(counts[i], want)
    b.close()
