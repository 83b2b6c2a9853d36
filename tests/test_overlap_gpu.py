"""Launches of one handle that overlap on the GPU: records of each complete, and of every later run."""
import numpy as np
import pytest
import torch

from optixsoltracedemos_gb300 import native, scenes

pytestmark = pytest.mark.gpu

SCENES = {"list": lambda: scenes.three_heliostats(num_rays=1),
          "grid": lambda: scenes.large_field(n_heliostats=300, sun=scenes.sun_vector(45.0, 20.0))}


@pytest.mark.parametrize("scene", SCENES)
@pytest.mark.parametrize("captured", [False, True])
def test_trace_async_beside_windows(gpu, oracle32, scene, captured):
    """trace_async on the caller's stream (called, or replayed from a graph) while windows are traced on the
    handle's own."""
    sc = SCENES[scene]()
    n, checked = 400_000, 20_000
    t = native.tracer_for(sc, seed=2, num_rays=n, record_ids=False)
    t.run()
    want, _ = t.copy_hits()
    oh, _ = oracle32.trace(sc.elements, sc.sun_dir, sc.sun_shape, sc.sun_param, count=checked, seed=2)
    np.testing.assert_array_equal(want[:checked], oh.astype(np.float32))
    want = torch.from_numpy(want).cuda()
    st = torch.cuda.Stream()
    graph = torch.cuda.CUDAGraph()
    if captured:
        with torch.cuda.graph(graph, stream=st):
            t.trace_async(st.cuda_stream)
    into = torch.empty(8, n, native.MAX_DEPTH, 4, device="cuda")
    own = torch.as_tensor(_Buffer(t, n), device="cuda")
    for _ in range(8):  # more launches than the handle has counters
        into.fill_(7.0)
        own.fill_(7.0)
        torch.cuda.synchronize()
        for k in range(8):
            if captured:
                with torch.cuda.stream(st):
                    graph.replay()
            else:
                t.trace_async(st.cuda_stream)
            t.trace_into(into[k].data_ptr(), None, 0, n)
        torch.cuda.synchronize()
        assert torch.equal(own, want) and all(torch.equal(w, want) for w in into)
    own.fill_(7.0)
    torch.cuda.synchronize()
    t.run()
    assert torch.equal(own, want)
    t.close()


class _Buffer:
    """View of a tracer's hit buffer."""

    def __init__(self, tracer, n):
        self.tracer = tracer
        self.__cuda_array_interface__ = {"data": (tracer.device_buffers()[0], False),
                                         "shape": (n, native.MAX_DEPTH, 4), "typestr": "<f4", "version": 3,
                                         "strides": None}
