"""Batches of more rays than the GPU has lanes (1,024 an SM), which trace one
ray a lane: the single-scene calls' results, bit for bit."""
import numpy as np
import pytest

from gridrt import scenes

pytestmark = pytest.mark.gpu


def _sizes(parts):
    """Ray counts of `parts` tasks, odd ones, above the resident lanes in all."""
    import torch
    lanes = 1024 * torch.cuda.get_device_properties(0).multi_processor_count
    return [lanes * 5 // 4 // parts + 37 * i + 1 for i in range(parts)]


def _rays(sc, n, seed, tmax=None):
    rays = scenes.random_rays(np.random.default_rng(seed), n, sc.verts.min(0), sc.verts.max(0))
    if tmax is not None:
        rays[:, 7] = tmax
    return rays


def _batch(gridlib, scs, tasks):
    """The scenes (uploaded) and (scene, mode, rays) tasks as a batch, and its outputs."""
    import torch
    t, outs = [], []
    for i, mode, rays in tasks:
        any_hit = mode == gridlib.RTG_MODE_ANY
        out = torch.full((len(rays), 1 if any_hit else 4), 77, dtype=torch.uint8 if any_hit else torch.int32,
                         device="cuda")
        t.append((i, mode, torch.from_numpy(rays).cuda(), len(rays), out))
        outs.append(out)
    return gridlib.Batch(scs, [4] * len(scs), t), t, outs


@pytest.mark.parametrize("refill", [0, 8])
def test_occlusion_with_a_tmax_that_is_not_a_number(gridlib, refill):
    """No hit lies before a tmax of NaN: not occluded, as for one scene."""
    sc = scenes.plane_and_debris(seed=7, quads=40, debris=3000)
    n, m = _sizes(2)
    seg = _rays(sc, n, 1, 0.4)
    seg[::3, 7] = np.nan
    s = gridlib.Scene(0)
    s.set_geometry(sc.verts, sc.idx)
    s.build(4)
    want = s.trace_any(seg)
    assert not want[::3].any() and (want == 1).any()
    b, _, outs = _batch(gridlib, [s], [(0, gridlib.RTG_MODE_ANY, seg), (0, gridlib.RTG_MODE_NEAREST, _rays(sc, m, 2))])
    b.set_tuning(refill=refill)
    b.build_async()
    b.trace_async()
    assert b.check() == 0
    assert np.array_equal(outs[0].cpu().numpy()[:, 0], want)


@pytest.mark.parametrize("cell_records,heavy,refill",
                         [(False, 0, 0), (True, 32, 0), (False, 4, 0), (True, 32, 8), (False, 4, 16), (False, 0, 1)])
def test_large_batch_equals_scene_traces(gridlib, cell_records, heavy, refill):
    """With and without cell-ordered records, hand-on and lane refill, against the
    scenes' one-lane walks without them.  Every ray in the soup meets lists above 4,
    so heavy = 4 also overfills the batch's queue of 65,536 rays."""
    kinds = [scenes.tiny_scene(3, 20_000), scenes.plane_and_debris(seed=5, quads=30, debris=9000),
             scenes.deforming_sphere(0), scenes.plane_and_debris(seed=6, quads=12, debris=300)]
    sizes = [75_001, 40_003, *_sizes(2)]
    scs, tasks, want = [], [], []
    for i, (sc, n) in enumerate(zip(kinds, sizes)):
        s = gridlib.Scene(0)
        s.set_geometry(sc.verts, sc.idx)
        s.set_tuning(lanes=1, heavy_cell=0, refill=0)
        s.build(4)
        rays, seg = _rays(sc, n, i), _rays(sc, n // 3 + 1, 50 + i, 0.5)
        cam = scenes.camera_rays(scenes.plane_and_debris_camera(64, 64))[:len(rays) // 4]
        rays[:len(cam)] = cam                                   # alike, then not
        want += [s.trace_nearest(rays).view(np.int32), s.trace_any(seg)]
        tasks += [(i, gridlib.RTG_MODE_NEAREST, rays), (i, gridlib.RTG_MODE_ANY, seg)]
        if cell_records and i % 2 == 0:
            s.set_tuning(cell_records=True)
        scs.append(s)
    b, _, outs = _batch(gridlib, scs, tasks)
    b.set_tuning(heavy_cell=heavy, heavy_lanes=4 if heavy == 4 else 8, refill=refill)
    for _ in range(2):
        b.build_async()
        b.trace_async()
        assert b.check() == 0
        for got, exp in zip(outs, want):
            assert np.array_equal(got.cpu().numpy().reshape(exp.shape), exp)
            got.fill_(77)
