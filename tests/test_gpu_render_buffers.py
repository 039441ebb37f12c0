"""Frames of rtg_render take their buffers from the scene's own pool: the pixels
and the ray counts must not depend on which frames came before (larger, smaller)
or run beside (other threads and streams of the same scene)."""
import threading

import numpy as np
import pytest

from gridrt import scenes

pytestmark = pytest.mark.gpu

SIZES = [(33, 17), (160, 120), (1, 1), (320, 200)]


def _frame(gridlib, s, normals, size, stream):
    import torch
    cam = scenes.plane_and_debris_camera(*size)
    mats = [gridlib.material(gridlib.RTG_MAT_PHONG, reflexion=0.35, opacity=0.6, refraction_index=1.3)]
    lights = [gridlib.point_light((2.0, 4.0, 2.0), (0.8, 0.8, 0.8), True)]
    with torch.cuda.stream(stream):
        rgb = torch.full((size[0] * size[1], 3), -1.0, dtype=torch.float32, device="cuda")
    rays = s.render(cam, normals, mats, lights, rgb, max_depth=3, stream=stream.cuda_stream)
    return rays, rgb.cpu().numpy()


def test_render_frames_of_one_scene_are_independent(gridlib):
    import torch
    sc = scenes.plane_and_debris()

    def scene():
        s = gridlib.Scene(0)
        s.set_geometry(sc.verts, sc.idx)
        s.build(4)
        return s

    normals = torch.tensor([[0.0, 1.0, 0.0]], device="cuda").repeat(sc.verts.shape[0], 1).contiguous()
    torch.cuda.synchronize()
    first = torch.cuda.Stream()
    want = {z: _frame(gridlib, scene(), normals, z, first) for z in SIZES}   # a new scene each
    assert want[(160, 120)][0] > 160 * 120
    s = scene()
    errors = []

    def run(order):
        try:
            stream = torch.cuda.Stream()
            for i in order:
                rays, rgb = _frame(gridlib, s, normals, SIZES[i], stream)
                assert rays == want[SIZES[i]][0]
                assert np.array_equal(rgb.view(np.int32), want[SIZES[i]][1].view(np.int32))
        except BaseException as e:   # reported by the main thread
            errors.append(e)

    threads = [threading.Thread(target=run, args=(o,)) for o in ([0, 3, 1, 2, 3], [3, 1, 0, 3, 2], [2, 1, 3, 0, 1])]
    for t in threads:
        t.start()
    for t in threads:
        t.join(120)
    assert not errors, errors[0]
