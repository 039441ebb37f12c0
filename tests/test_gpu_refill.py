"""Ray arrays traced one ray a lane: 32 consecutive rays that are alike are
traced together, others refilled lane by lane; whatever the mix, the results are
those of tracing 32 rays at a time, bit for bit."""
import numpy as np
import pytest

from gridrt import scenes

pytestmark = pytest.mark.gpu


def _mix(kind, n):
    """n rays: camera rays, random ones, or runs of either that end inside a
    group of 32; some slots hold no ray (tmax < 0)."""
    cam = scenes.camera_rays(scenes.plane_and_debris_camera(256, 256), "morton8")[:n]
    rnd = scenes.random_rays(np.random.default_rng(5), n, (-1, 0, -1), (1, 1, 1))
    run = (np.arange(n) // 77) % 2 == 0
    rays = {"camera": cam, "random": rnd, "runs": np.where(run[:, None], cam, rnd),
            "camera first": np.concatenate([cam[:n // 2], rnd[n // 2:]])}[kind].copy()
    seg = rays.copy()
    seg[:, 7] = 0.7
    seg[::13, 7] = -1.0
    return rays, seg


@pytest.mark.parametrize("kind", ["camera", "random", "runs", "camera first"])
@pytest.mark.parametrize("n", [1, 31, 33, 4097, 65536])
def test_arrays_alike_or_not(gridlib, kind, n):
    import torch
    sc = scenes.plane_and_debris(quads=64, debris=8000)
    s = gridlib.Scene(0)
    s.set_geometry(sc.verts, sc.idx)
    s.set_tuning(lanes=1, refill=0)
    s.build(4)
    rays, seg = _mix(kind, n)
    want = s.trace_nearest(rays).view(np.int32), s.trace_any(seg)
    for refill, heavy in ((1, 32), (8, 32), (8, 2), (32, 0)):
        s.set_tuning(refill=refill, heavy_cell=heavy)
        assert np.array_equal(s.trace_nearest(rays).view(np.int32), want[0]), (refill, heavy)
        assert np.array_equal(s.trace_any(seg), want[1]), (refill, heavy)
    # the same rays as tasks of a batch large enough for one ray a lane
    s.set_tuning(heavy_cell=32)
    lanes = 1024 * torch.cuda.get_device_properties(0).multi_processor_count
    pad = torch.from_numpy(_mix("camera", 65536)[0]).cuda().repeat(lanes * 5 // 4 // 65536 + 1, 1)
    outs = [torch.full((n, 4), 7, dtype=torch.int32, device="cuda"),
            torch.full((n,), 7, dtype=torch.uint8, device="cuda"),
            torch.zeros((len(pad), 4), dtype=torch.int32, device="cuda")]
    b = gridlib.Batch([s], [4], [(0, 0, torch.from_numpy(rays).cuda(), n, outs[0]),
                                 (0, 1, torch.from_numpy(seg).cuda(), n, outs[1]),
                                 (0, 0, pad, len(pad), outs[2])])
    b.build_async()
    b.trace_async()
    assert b.check() == 0
    assert np.array_equal(outs[0].cpu().numpy(), want[0])
    assert np.array_equal(outs[1].cpu().numpy(), want[1])
