"""Images that a small mesh fills are traced one ray a lane where that is the
faster, images that it does not by groups of lanes; the results are the same
bits."""
import pytest

import timing
from gridrt import scenes

pytestmark = pytest.mark.gpu


def _camera(width, height, eye=(1.6, 1.2, 2.4)):
    return scenes.look_at_camera(eye, (0.0, 0.0, 0.0), (0.0, 1.0, 0.0), 60.0, width, height)


def _lanes():
    import torch
    return 1024 * torch.cuda.get_device_properties(0).multi_processor_count


@pytest.mark.parametrize("lat,k", [(24, 4), (80, 8)])
@pytest.mark.parametrize("call", ["frame", "camera"])
@pytest.mark.parametrize("shape,eye", [("tall", (1.6, 1.2, 2.4)), ("square", (1.6, 1.2, 2.4)), ("square", (0.3, 0.1, 0.2))])
def test_results_do_not_depend_on_the_lanes(gridlib, lat, k, call, shape, eye):
    """Around every limit of a launch's size; also from inside the scene's box."""
    import torch
    v, i, _ = scenes.sphere_mesh(lat, 2 * lat + 1)
    s = gridlib.Scene(0)
    s.set_geometry(v, i)
    s.build(k)
    for part in (0.7, 1.0, 1.24, 1.26, 1.49, 1.51, 1.74, 1.76):
        n = part * _lanes()
        width = int((n / 4) ** 0.5) if shape == "tall" else int(n ** 0.5)
        cam = _camera(width, int(n / width), eye)
        m = cam.width * cam.height
        got = []
        for lanes in (-1, 1):
            s.set_tuning(lanes=lanes)
            hits = torch.zeros((m, 4), dtype=torch.int32, device="cuda")
            occ = torch.full((m,), 7, dtype=torch.uint8, device="cuda")
            sr = torch.zeros((m, 8), dtype=torch.float32, device="cuda")
            if call == "frame":
                s.trace_frame_device(cam, scenes.SPHERE_LIGHT, hits, occ, sr)
            else:
                s.trace_camera_device(cam, hits, scenes.SPHERE_LIGHT, sr)
            torch.cuda.synchronize()
            got.append((hits, occ, sr.view(torch.int32)))
        assert (got[0][0][:, 0] >= 0).any()
        for a, b in zip(*got):
            assert torch.equal(a, b), (part, shape)
    s.close()


@pytest.mark.parametrize("call,scene", [("frame", 24), ("frame", 80), ("camera", "debris")])
def test_a_small_mesh_that_fills_the_image(gridlib, call, scene):
    """As fast as with lanes = 1 (on 152 SMs: frames of 2,352 triangles 94 us, of
    25,760 134, camera rays of plane and debris 69; by 8 lanes a ray 117, 197 and
    87 us, and some 15 more in each call that is waited for)."""
    import torch
    if scene == "debris":
        sc = scenes.plane_and_debris(quads=22, debris=1032)
        v, i, k, light, eye = sc.verts, sc.idx, 8, scenes.PLANE_LIGHT, (0.0, 1.5, 3.0)
    else:
        v, i, _ = scenes.sphere_mesh(scene, 2 * scene + 1)
        k, light, eye = 4, scenes.SPHERE_LIGHT, (1.6, 1.2, 2.4)
    s = gridlib.Scene(0)
    s.set_geometry(v, i)
    s.build(k)
    n = 1.68 * _lanes()
    cam = _camera(int((n / 4) ** 0.5), int(n / int((n / 4) ** 0.5)), eye)
    m = cam.width * cam.height
    hits = torch.zeros((m, 4), dtype=torch.int32, device="cuda")
    occ = torch.zeros(m, dtype=torch.uint8, device="cuda")
    sr = torch.zeros((m, 8), dtype=torch.float32, device="cuda")

    def go(s):
        if call == "frame":
            s.trace_frame_device(cam, light, hits, occ, sr)
        else:
            s.trace_camera_device(cam, hits, light, sr)

    one = gridlib.Scene(0)
    one.set_geometry(v, i)
    one.set_tuning(lanes=1)
    one.build(k)
    assert timing.ratio(lambda: go(s), lambda: go(one), 1.12) < 1.12
