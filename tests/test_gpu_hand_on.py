"""Random rays of a launch a little larger than the GPU's resident lanes: those that
meet many triangles are handed on early, so that the launch does not wait for
them; the results are those of tracing every ray to its end."""
import numpy as np
import pytest

import timing
from gridrt import scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", ["nearest", "any"])
def test_random_rays_beyond_the_resident_lanes(gridlib, mode):
    """As fast as when told to hand rays on after 128 tests: plane and debris of
    2,000 triangles, 102 us for 1.3 rays a lane and 127 for as many segments
    (152 SMs); after 256 tests 120 and 148."""
    import torch
    sc = scenes.plane_and_debris(quads=22, debris=1032)
    n = 1024 * torch.cuda.get_device_properties(0).multi_processor_count * 13 // 10
    rays = scenes.random_rays(np.random.default_rng(3), n, sc.verts.min(0), sc.verts.max(0))
    if mode == "any":
        rays[:, 7] = 0.7
    rays = torch.from_numpy(rays).cuda()
    s, early = gridlib.Scene(0), gridlib.Scene(0)
    for x in (s, early):
        x.set_geometry(sc.verts, sc.idx)
        x.build(8)
        x.set_tuning(lanes=1)
    early.set_tuning(heavy_cell=16)          # 8 thresholds: 128 tests
    outs = [torch.full((n, 4) if mode == "nearest" else (n,), x,
                       dtype=torch.int32 if mode == "nearest" else torch.uint8, device="cuda") for x in (7, 8, 9)]

    def trace(x, out):
        return x.trace_nearest_device(rays, n, out) if mode == "nearest" else x.trace_any_device(rays, n, out)

    slower = timing.ratio(lambda: trace(s, outs[0]), lambda: trace(early, outs[1]), 1.08)
    early.set_tuning(heavy_cell=0)
    trace(early, outs[2])
    torch.cuda.synchronize()
    assert torch.equal(outs[0], outs[2]) and torch.equal(outs[1], outs[2])
    if mode == "nearest":
        assert slower < 1.08


@pytest.mark.parametrize("heavy", [1, 4, 16, 64])
def test_hand_on_of_the_one_lane_walk(gridlib, heavy):
    """Rays handed on by one lane give the bits of the walk that hands none on, for
    frames, camera rays and arrays; small thresholds also overfill the queue."""
    import torch
    sc = scenes.deforming_sphere(2)
    cam = scenes.deforming_sphere_camera(512, 512)
    n = 512 * 512
    rays = scenes.random_rays(np.random.default_rng(11), 120_000, (-1.2, -1.2, -1.2), (1.2, 1.2, 1.2))
    seg = rays.copy()
    seg[:, 7] = 0.5
    s = gridlib.Scene(0)
    s.set_geometry(sc.verts, sc.idx)
    s.set_tuning(lanes=1)

    def results(order):
        hits = torch.zeros((n, 4), dtype=torch.int32, device="cuda")
        occ = torch.full((n,), 7, dtype=torch.uint8, device="cuda")
        sr = torch.zeros((n, 8), dtype=torch.float32, device="cuda")
        s.trace_frame_device(cam, scenes.SPHERE_LIGHT, hits, occ, sr, order=order)
        hits2, sr2 = torch.zeros_like(hits), torch.zeros_like(sr)
        s.trace_camera_device(cam, hits2, scenes.SPHERE_LIGHT, sr2, order=order)
        torch.cuda.synchronize()
        out = [x.cpu().numpy() for x in (hits, occ, sr, hits2, sr2)]
        return [x.view(np.uint32) if x.dtype == np.float32 else x for x in out] + [
            s.trace_nearest(rays).view(np.int32), s.trace_any(seg)]

    s.set_tuning(heavy_cell=0, refill=0)
    s.build(8)
    want = {order: results(order) for order in ("scanline", "morton8")}
    for records, lanes, refill in ((False, 8, 0), (True, 4, 16), (True, 16, 1), (False, 32, 8)):
        s.set_tuning(heavy_cell=heavy, cell_records=records, heavy_lanes=lanes, refill=refill)
        s.build(8)
        for order in want:
            for a, b in zip(want[order], results(order)):
                assert np.array_equal(a, b), (records, lanes, refill, order)
    s.close()
