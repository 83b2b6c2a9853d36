"""Record and element-id rows of field launches (grid and BVH), written by the warp from shared memory in
coherent order: windows that end inside a warp, a tile and each block size of the order (55,296 rays,
331,776, 1,990,656), with and without ids, equal to the oracle; nothing is written past the window."""
import numpy as np
import pytest
import torch

from optixsoltracedemos_gb300 import native, scenes

pytestmark = pytest.mark.gpu

B3, B2, B1 = 55_296, 331_776, 1_990_656
COUNTS = [1, 31, 33, 127, 129, B3 - 1, B3, B3 + 1, 2 * B3 + 130, B2 - 1, B2 + B3 + 37, B1 + B3 + 65]


@pytest.mark.parametrize("count", COUNTS)
@pytest.mark.parametrize("accel", [native.ACCEL_GRID, native.ACCEL_BVH])
def test_dense_rows_equal_oracle(gpu, oracle32, count, accel):
    sc = scenes.large_field(n_heliostats=40, sun=scenes.sun_vector(50.0, -30.0))
    first = 12_345
    # past 10^5 rays the oracle checks both ends
    spans = [(0, count)] if count < 100_000 else [(0, 20_000), (count - 20_000, count)]
    t = native.tracer_for(sc, seed=3, num_rays=1, accel=accel)
    for with_ids in (True, False):
        hits = torch.full((count + 1, native.MAX_DEPTH, 4), 7.0, device="cuda")
        ids = torch.full((count + 1, native.MAX_DEPTH), 7, device="cuda", dtype=torch.int32)
        t.trace_into(hits.data_ptr(), ids.data_ptr() if with_ids else None, first, count)
        torch.cuda.synchronize()
        assert (hits[count] == 7.0).all() and (ids[count] == 7).all()
        assert with_ids or (ids == 7).all()
        for a, b in spans:
            oh, oi = oracle32.trace(sc.elements, sc.sun_dir, sc.sun_shape, sc.sun_param, first_ray=first + a,
                                    count=b - a, seed=3)
            np.testing.assert_array_equal(hits[a:b].cpu().numpy(), oh.astype(np.float32))
            if with_ids:
                np.testing.assert_array_equal(ids[a:b].cpu().numpy().view(np.uint32), oi)
        if count >= 100_000:  # between the ends: every row has its sun-plane point and no leftover
            assert not (hits[:count] == 7.0).all(dim=2).any()
    t.close()


@pytest.mark.parametrize("count", [B3 + 77, B2 + 33, B1 + B2 + B3 + 65])
@pytest.mark.parametrize("accel", [native.ACCEL_GRID, native.ACCEL_BVH])
def test_every_row_of_coherent_blocks(gpu, count, accel):
    """Every row of launches of each block size equals that of the same rays in windows too short for a block
    (identity order, which the oracle checks above): each lane's record in its own row."""
    sc = scenes.large_field(n_heliostats=40, sun=scenes.sun_vector(50.0, -30.0))
    first, window = 12_345, 50_000
    t = native.tracer_for(sc, seed=3, num_rays=1, accel=accel)
    want = torch.full((count, native.MAX_DEPTH, 4), 7.0, device="cuda")
    want_ids = torch.full((count, native.MAX_DEPTH), 7, device="cuda", dtype=torch.int32)
    torch.cuda.synchronize()
    for a in range(0, count, window):
        t.trace_into(want[a:].data_ptr(), want_ids[a:].data_ptr(), first + a, min(window, count - a))
    torch.cuda.synchronize()
    assert (want[:, 0, 0] == 0).all() and (want[:, 1:, 0] == 1).any()
    for with_ids in (True, False):
        hits = torch.full_like(want, 7.0)
        ids = torch.full_like(want_ids, 7)
        torch.cuda.synchronize()
        t.trace_into(hits.data_ptr(), ids.data_ptr() if with_ids else None, first, count)
        torch.cuda.synchronize()
        assert torch.equal(hits, want)
        if with_ids:
            assert torch.equal(ids, want_ids)
    t.close()
