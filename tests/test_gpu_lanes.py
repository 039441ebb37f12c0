"""Launches too small to fill the GPU trace each ray with a group of lanes: the
hits, shadow rays and occlusion of every group size are the one-lane walk's,
bit for bit, at the launch sizes where the group size changes."""
import numpy as np
import pytest

from gridrt import scenes

pytestmark = pytest.mark.gpu


def _rays(sc, n, seed, tmax=None):
    rays = scenes.random_rays(np.random.default_rng(seed), n, sc.verts.min(0), sc.verts.max(0))
    if tmax is not None:
        rays[:, 7] = tmax
    return rays


def _edges():
    """Ray counts around each change of the group size (1,024 lanes an SM)."""
    import torch
    lanes = 1024 * torch.cuda.get_device_properties(0).multi_processor_count
    return [1, 31, 33, lanes // 8, lanes // 8 + 1, lanes // 2, lanes // 2 + 1, lanes * 5 // 4, lanes * 5 // 4 + 1]


@pytest.mark.parametrize("name", ["plane", "cluster", "one"])
def test_ray_arrays_by_groups_equal_one_lane(gridlib, name):
    sc, k = {"plane": lambda: (scenes.plane_and_debris(quads=64, debris=8000), 4),
             "cluster": lambda: (scenes.skewed_density(n=1 << 16), 4),    # lists above 2,048: the block pass
             "one": lambda: (scenes.tiny_scene(3, 1), 6)}[name]()
    s = gridlib.Scene(0)
    s.set_geometry(sc.verts, sc.idx)
    s.build(k)
    for i, n in enumerate(_edges()):
        rays, seg = _rays(sc, n, i), _rays(sc, n, 100 + i, 0.4)
        got = s.trace_nearest(rays).view(np.int32), s.trace_any(seg)
        s.set_tuning(lanes=1)
        want = s.trace_nearest(rays).view(np.int32), s.trace_any(seg)
        s.close()
        s = gridlib.Scene(0)
        s.set_geometry(sc.verts, sc.idx)
        s.build(k)
        assert np.array_equal(got[0], want[0]), (name, n)
        assert np.array_equal(got[1], want[1]), (name, n)


@pytest.mark.parametrize("side", [(8, 8), (136, 136), (272, 272), (280, 288), (512, 528), (520, 528), (552, 560), (568, 560)])
def test_frames_by_groups_equal_one_lane(gridlib, side):
    import torch
    sc = scenes.deforming_sphere(3)
    cam = scenes.deforming_sphere_camera(*side)
    n = side[0] * side[1]
    out = []
    for lanes, records in ((None, False), (None, True), (1, False)):
        s = gridlib.Scene(0)
        s.set_tuning(lanes=lanes, cell_records=records)
        s.set_geometry(sc.verts, sc.idx)
        s.build(8)
        hits = torch.zeros((n, 4), dtype=torch.int32, device="cuda")
        occ = torch.zeros(n, dtype=torch.uint8, device="cuda")
        sr = torch.zeros((n, 8), dtype=torch.float32, device="cuda")
        s.trace_frame_device(cam, scenes.SPHERE_LIGHT, hits, occ, sr, order="morton8")
        torch.cuda.synchronize()
        out.append((hits.cpu().numpy(), occ.cpu().numpy(), sr.cpu().numpy().view(np.uint32)))
        s.close()
    for got in out[:2]:
        for a, b in zip(got, out[2]):
            assert np.array_equal(a, b), side


@pytest.mark.parametrize("rays", [1, 700, 9000, 40000])
def test_small_batches_by_groups_equal_single_scenes(gridlib, rays):
    import torch
    scs, tasks, want = [], [], []
    for i in range(3):
        sc = scenes.plane_and_debris(seed=50 + i, quads=20, debris=500 * (i + 1))
        s = gridlib.Scene(0)
        s.set_geometry(sc.verts, sc.idx)
        s.build(4)
        s.set_tuning(lanes=1)
        r, g = _rays(sc, rays + 7 * i, i), _rays(sc, rays + 3, 10 + i, 0.3)
        want.append((s.trace_nearest(r).view(np.int32), s.trace_any(g)))
        scs.append(s)
        for mode, x, kind, width in ((0, r, torch.int32, 4), (1, g, torch.uint8, 1)):
            out = torch.full((len(x), width), 77, dtype=kind, device="cuda")
            tasks.append((i, mode, torch.from_numpy(x).cuda(), len(x), out))
    b = gridlib.Batch(scs, [4, 4, 4], tasks)
    b.build_async()
    b.trace_async()
    assert b.check() == 0
    for i in range(3):
        assert np.array_equal(tasks[2 * i][4].cpu().numpy(), want[i][0]), i
        assert np.array_equal(tasks[2 * i + 1][4].cpu().numpy()[:, 0], want[i][1]), i
