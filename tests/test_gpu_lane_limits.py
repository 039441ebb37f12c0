"""The launch sizes on both sides of every limit of the lanes per ray: the numbers of
launches tell the variants apart (one lane a ray has a pass behind it, groups in a
scene of short lists none), and the results are one lane's, bit for bit."""
import numpy as np
import pytest

from gridrt import scenes

pytestmark = pytest.mark.gpu


def _lanes():
    import torch
    return 1024 * torch.cuda.get_device_properties(0).multi_processor_count


def _rays(sc, n, seed, tmax=None):
    rays = scenes.random_rays(np.random.default_rng(seed), n, sc.verts.min(0), sc.verts.max(0))
    if tmax is not None:
        rays[:, 7] = tmax
    return rays


def _scene(gridlib, sc, k=4):
    s = gridlib.Scene(0)
    s.set_geometry(sc.verts, sc.idx)
    s.build(k)
    return s


def _counted(gridlib, call):
    before = gridlib.kernel_launches()
    out = call()
    return gridlib.kernel_launches() - before, out


@pytest.mark.parametrize("mode", ["nearest", "any"])
def test_arrays_at_the_limits(gridlib, mode):
    R = _lanes()
    last = R if mode == "nearest" else 3 * R // 4        # the largest launch of 8 lanes a ray
    sc = scenes.plane_and_debris(quads=64, debris=8000)
    s = _scene(gridlib, sc)
    off, _ = s.download()
    assert np.diff(off).max() <= 32 * 4                  # 8 lanes deal every list themselves
    for n, launches in ((R // 8, 1), (R // 8 + 1, 1), (R // 2, 1), (R // 2 + 1, 1), (last - 31, 1), (last, 1),
                        (last + 1, 2), (last + 33, 2)):
        rays = _rays(sc, n, n % 97, None if mode == "nearest" else 0.4)
        trace = s.trace_nearest if mode == "nearest" else s.trace_any
        s.set_tuning(lanes=-1)
        count, got = _counted(gridlib, lambda: trace(rays))
        assert count == launches, n
        s.set_tuning(lanes=1)
        count, want = _counted(gridlib, lambda: trace(rays))
        assert count == 2 and np.array_equal(got.view(np.uint8), want.view(np.uint8)), n
    s.close()


@pytest.mark.parametrize("call", ["frame", "camera"])
def test_images_at_the_limits(gridlib, call):
    import torch
    R = _lanes()
    sc = scenes.plane_and_debris(quads=160, debris=60_000)    # more triangles than a small mesh
    s = _scene(gridlib, sc)
    off, _ = s.download()
    assert np.diff(off).max() <= 32 * 4
    for n, launches in ((R // 8, 1), (R // 8 + 64, 1), (R // 2, 1), (R // 2 + 64, 1), (7 * R // 4, 1),
                        (7 * R // 4 + 64, 2)):
        cam = scenes.plane_and_debris_camera(64, n // 64)
        n = 64 * (n // 64)
        got = []
        for lanes in (-1, 1):
            s.set_tuning(lanes=lanes)
            hits = torch.zeros((n, 4), dtype=torch.int32, device="cuda")
            occ = torch.full((n,), 7, dtype=torch.uint8, device="cuda")
            sr = torch.zeros((n, 8), dtype=torch.float32, device="cuda")
            count, _ = _counted(gridlib, lambda: s.trace_frame_device(cam, scenes.PLANE_LIGHT, hits, occ, sr)
                                if call == "frame" else s.trace_camera_device(cam, hits, scenes.PLANE_LIGHT, sr))
            torch.cuda.synchronize()
            got.append((hits, occ, sr.view(torch.int32)))
            assert count == (launches if lanes < 0 else 2), (n, lanes)
        for a, b in zip(*got):
            assert torch.equal(a, b), n
    s.close()


@pytest.mark.parametrize("over", [0, 32])
def test_batches_at_the_limit(gridlib, over):
    """Totals of padded rays: the resident lanes, and one group of 32 more."""
    import torch
    total = _lanes() + over
    scs = [_scene(gridlib, scenes.plane_and_debris(seed=60 + i, quads=20, debris=700 * (i + 1))) for i in range(2)]
    first = total // 2 // 32 * 32
    tasks, want = [], []
    for i, n in enumerate((first - 13, total - first - 7)):   # each padded to a multiple of 32
        rays = _rays(scenes.plane_and_debris(seed=60 + i, quads=20, debris=700 * (i + 1)), n, i)
        scs[i].set_tuning(lanes=1)
        want.append(scs[i].trace_nearest(rays).view(np.int32))
        out = torch.full((n, 4), 77, dtype=torch.int32, device="cuda")
        tasks.append((i, gridlib.RTG_MODE_NEAREST, torch.from_numpy(rays).cuda(), n, out))
    b = gridlib.Batch(scs, [4, 4], tasks)
    b.build_async()
    count, _ = _counted(gridlib, b.trace_async)
    assert count == (2 if over else 1)
    assert b.check() == 0
    for t, w in zip(tasks, want):
        assert np.array_equal(t[4].cpu().numpy(), w)
    b.close()
