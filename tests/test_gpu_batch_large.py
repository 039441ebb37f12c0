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
