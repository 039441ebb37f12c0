"""Render buffers kept between frames: 1 GiB a device at most, of however many
scenes; the scenes that rendered least recently give theirs back first, and a
scene's go with it."""
import gc

import numpy as np
import pytest

from gridrt import scenes

pytestmark = pytest.mark.gpu

KEEP = 1 << 30


def test_kept_render_buffers_are_bounded(gridlib):
    import torch
    sc = scenes.plane_and_debris()
    cam = scenes.plane_and_debris_camera(1280, 960)
    n = cam.width * cam.height
    normals = torch.tensor([[0.0, 1.0, 0.0]], device="cuda").repeat(sc.verts.shape[0], 1).contiguous()
    mats = [gridlib.material(gridlib.RTG_MAT_PHONG, reflexion=0.35, opacity=0.6, refraction_index=1.3)]
    lights = [gridlib.point_light((2.0, 4.0, 2.0), (0.8, 0.8, 0.8), True)]
    stream = torch.cuda.Stream()

    def scene():
        s = gridlib.Scene(0)
        s.set_geometry(sc.verts, sc.idx)
        s.build(4)
        return s

    def free():
        torch.cuda.synchronize()
        return torch.cuda.mem_get_info()[0]

    rgb = torch.zeros((n, 3), dtype=torch.float32, device="cuda")

    def frame(s):
        s.render(cam, normals, mats, lights, rgb, max_depth=3, stream=stream.cuda_stream)
        return rgb.cpu().numpy().view(np.int32)

    gc.collect()                                       # scenes of other tests
    warm = scene()
    want = frame(warm)                                 # modules loaded
    warm.close()
    many = [scene() for _ in range(5)]
    start = free()
    assert np.array_equal(frame(many[0]), want)
    one = start - free()
    assert one > KEEP // 4                             # a frame's levels are kept, and five exceed the bound
    for s in many[1:]:
        assert np.array_equal(frame(s), want)
        assert start - free() <= KEEP
    assert np.array_equal(frame(many[0]), want)        # it had given its own back
    assert start - free() <= KEEP
    kept = start - free()
    before = free()
    for s in many:
        s.close()
    assert free() - before >= kept                     # (and the scenes' own buffers)
