"""The shadow rays a camera pass writes, given as an array to the occlusion call:
most slots of the sphere's image hold none, and its rim is in every row, yet its
neighbouring rays are alike and are traced as such."""
import pytest

import timing
from gridrt import scenes

pytestmark = pytest.mark.gpu


def _pair(gridlib, verts, idx):
    """The scene at one lane a ray, and the same with every 32 rays traced together."""
    out = []
    for refill in (None, 0):
        s = gridlib.Scene(0)
        s.set_geometry(verts, idx)
        s.set_tuning(lanes=1, refill=refill)
        s.build(4)
        out.append(s)
    return out


@pytest.mark.parametrize("order", ["scanline", "morton8"])
def test_shadow_rays_of_an_image(gridlib, order):
    """As fast as with refill 0, which traces every 32 consecutive rays together:
    95 us on 152 SMs.  Taken for rays that differ, they took 131 (scanline) and
    124 us; the bound lies between."""
    import torch
    sc = scenes.deforming_sphere(3)
    cam = scenes.deforming_sphere_camera(640, 480)
    n = cam.width * cam.height
    s, whole = _pair(gridlib, sc.verts, sc.idx)
    hits = torch.zeros((n, 4), dtype=torch.int32, device="cuda")
    rays = torch.zeros((n, 8), dtype=torch.float32, device="cuda")
    s.trace_camera_device(cam, hits, scenes.SPHERE_LIGHT, rays, order=order)
    torch.cuda.synchronize()
    assert (rays[:, 7] < 0).float().mean() > 0.5
    got, want = torch.zeros(n, dtype=torch.uint8, device="cuda"), torch.ones(n, dtype=torch.uint8, device="cuda")
    slower = timing.ratio(lambda: s.trace_any_device(rays, n, got), lambda: whole.trace_any_device(rays, n, want), 1.15)
    assert torch.equal(got, want)
    assert slower < 1.15


def test_camera_rays_whose_rows_end_inside_a_chunk(gridlib):
    """As fast as with refill 0: of the sphere of 2,352 triangles 72 us at
    540 x 540 on 152 SMs, of 25,760 triangles 116 to 141; taken for rays that
    differ, 100 and 167, and some 15 more in each call that is waited for."""
    import torch
    for lat in (24, 80):
        v, i, _ = scenes.sphere_mesh(lat, 2 * lat + 1)
        s, whole = _pair(gridlib, v, i)
        rays = torch.from_numpy(scenes.camera_rays(scenes.deforming_sphere_camera(540, 540))).cuda()
        got, want = (torch.full((len(rays), 4), x, dtype=torch.int32, device="cuda") for x in (7, 8))
        slower = timing.ratio(lambda: s.trace_nearest_device(rays, len(rays), got),
                              lambda: whole.trace_nearest_device(rays, len(rays), want), 1.12)
        assert torch.equal(got, want)
        assert slower < 1.12, lat


def test_shadow_rays_of_a_small_image(gridlib):
    """Rays that are half alike, in a launch of a few chunks a warp: as fast as
    with refill 0 (plane and debris of 5,000 triangles, 512^2: 58 us; lane by
    lane 70, and some 15 more in each call that is waited for)."""
    import torch
    sc = scenes.plane_and_debris(quads=35, debris=2550)
    cam = scenes.look_at_camera((0.0, 1.5, 3.0), (0.0, 0.3, 0.0), (0.0, 1.0, 0.0), 60.0, 512, 512)
    n = cam.width * cam.height
    s, whole = _pair(gridlib, sc.verts, sc.idx)
    hits = torch.zeros((n, 4), dtype=torch.int32, device="cuda")
    rays = torch.zeros((n, 8), dtype=torch.float32, device="cuda")
    s.trace_camera_device(cam, hits, scenes.PLANE_LIGHT, rays)
    got, want = torch.zeros(n, dtype=torch.uint8, device="cuda"), torch.ones(n, dtype=torch.uint8, device="cuda")
    slower = timing.ratio(lambda: s.trace_any_device(rays, n, got), lambda: whole.trace_any_device(rays, n, want), 1.08)
    assert torch.equal(got, want)
    assert slower < 1.08
