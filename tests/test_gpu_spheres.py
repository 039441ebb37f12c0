"""Scenes with lists above 4,096 entries, whose synchronous builds also write
the entries' bounding spheres: the builds give the oracle's grid, and a trace
tests the present lists, whoever built them last."""
import numpy as np
import pytest

from gridrt import scenes
from test_gpu_crowded import _crowd
from test_zz_no_alloc import _resolution_is_ambiguous

pytestmark = pytest.mark.gpu


def _ambiguous_crowd(k=4, n=200, crowd=9000):
    """A soup of n triangles and a crowd in one cell, with one triangle whose
    extent puts the resolution on a powf ulp boundary."""
    rng = np.random.default_rng(5)
    cent = rng.uniform(0.05, 0.95, size=(n, 1, 3))
    soup = cent + rng.uniform(-0.03, 0.03, size=(n, 3, 3))
    dense = np.array([0.31, 0.57, 0.43]) + rng.uniform(-5e-4, 5e-4, size=(crowd, 3, 3))
    verts = np.concatenate([soup, dense]).astype(np.float32).reshape(-1, 3)
    ends = np.stack([verts.min(0), verts.max(0)])       # all that the resolution takes from them
    for i in range(2_000_000):
        last = np.array([[0, 0, 0], [0.5, 1, 1], [1.0 + 1e-6 * i, 0.5, 0.5]], np.float32)
        if _resolution_is_ambiguous(np.concatenate([ends, last]), n + crowd + 1, k):
            v = np.concatenate([verts, last])
            return v, np.arange(len(v), dtype=np.int32).reshape(-1, 3)
    raise AssertionError("no ambiguous extent found")


def test_crowded_scene_of_host_resolved_parameters(gridlib, oracle):
    """The first build of a crowded scene makes room for the spheres and builds
    once more, also when its resolution was decided on the host."""
    verts, idx = _ambiguous_crowd()
    g = oracle.Grid(verts, idx, 4)
    assert np.diff(g.offsets).max() > 4096
    s = gridlib.Scene(0)
    s.set_geometry(verts, idx)
    for _ in range(2):
        s.build(4)
        off, ids = s.download()
        assert np.array_equal(off, g.offsets) and np.array_equal(ids, g.ids)
    s.close()


def _reversed_crowd(sc):
    """The same triangles, the crowd's in the reverse order: the same lists, but
    another triangle at every place of them."""
    v = sc.verts.reshape(-1, 3, 3).copy()
    v[60:] = v[60:][::-1]
    return v.reshape(-1, 3)


def _crowd_rays(sc, n=3000):
    mid = sc.verts.reshape(-1, 3, 3)[60:].mean(axis=(0, 1))
    rng = np.random.default_rng(n)
    rays = scenes.random_rays(rng, n, mid - 4, mid + 4)
    rays[:, 4:7] = (mid + rng.normal(size=(n, 3)) * 0.01 - rays[:, 0:3]).astype(np.float32)
    return rays


def _hits_of(gridlib, verts, idx, rays):
    s = gridlib.Scene(0)
    s.set_geometry(verts, idx)
    s.build(1)
    s.set_tuning(heavy_cell=0, lanes=2)      # every entry tested
    hits = s.trace_nearest(rays).view(np.int32)
    s.close()
    return hits


@pytest.fixture()
def moved(gridlib):
    sc = _crowd("tiny", 9000)
    rays = _crowd_rays(sc)
    verts = _reversed_crowd(sc)
    before, after = _hits_of(gridlib, sc.verts, sc.idx, rays), _hits_of(gridlib, verts, sc.idx, rays)
    assert (before[:, 0] != after[:, 0]).mean() > 0.2
    return sc, verts, rays, before, after


def _capture(stream, call):
    import torch
    call()                                   # tables and modules before the capture
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=stream):
        call()
    return g


def test_replayed_batch_build_of_a_scene_with_spheres(gridlib, moved):
    """A captured batch rebuilds a scene whose own build had written spheres."""
    import torch
    sc, verts, rays, before, after = moved
    s = gridlib.Scene(0)
    s.set_geometry(sc.verts, sc.idx)
    out = torch.zeros((64, 4), dtype=torch.int32, device="cuda")
    b = gridlib.Batch([s], [1], [(0, gridlib.RTG_MODE_NEAREST, torch.from_numpy(rays[:64]).cuda(), 64, out)])
    stream = torch.cuda.Stream()

    def step():
        b.build_async(stream.cuda_stream)
        b.trace_async(stream.cuda_stream)

    g = _capture(stream, step)
    s.build(1)
    assert np.array_equal(s.trace_nearest(rays).view(np.int32), before)
    s.update_vertices(verts, len(verts), False)
    torch.cuda.synchronize()
    g.replay()
    torch.cuda.synchronize()
    assert b.check() == 0
    assert np.array_equal(out.cpu().numpy(), after[:64])
    assert np.array_equal(s.trace_nearest(rays).view(np.int32), after)


def test_replayed_trace_of_a_scene_a_batch_rebuilt(gridlib, moved):
    """A captured trace of a scene with spheres, after a batch has rebuilt it;
    and again once its own build has written them anew."""
    import torch
    sc, verts, rays, before, after = moved
    s = gridlib.Scene(0)
    s.set_geometry(sc.verts, sc.idx)
    b = gridlib.Batch([s], [1], [])
    s.build(1)
    d_rays, hits = torch.from_numpy(rays).cuda(), torch.zeros((len(rays), 4), dtype=torch.int32, device="cuda")
    stream = torch.cuda.Stream()
    g = _capture(stream, lambda: s.trace_nearest_device(d_rays, len(rays), hits, stream=stream.cuda_stream))

    def replay():
        hits.zero_()
        torch.cuda.synchronize()
        g.replay()
        torch.cuda.synchronize()
        return hits.cpu().numpy()

    assert np.array_equal(replay(), before)
    s.update_vertices(verts, len(verts), False)
    torch.cuda.synchronize()
    b.build_async()
    assert b.check() == 0
    assert np.array_equal(replay(), after)
    s.build(1)
    assert np.array_equal(replay(), after)
    s.update_vertices(sc.verts, len(sc.verts), False)
    s.build_async(1)
    torch.cuda.synchronize()
    assert np.array_equal(replay(), before)


def _launches(gridlib, call):
    before = gridlib.kernel_launches()
    call()
    return gridlib.kernel_launches() - before


def _reserved(gridlib, verts, idx, k):
    """A scene with room for its grid, so that its first build needs no retry."""
    s = gridlib.Scene(0)
    s.set_geometry(verts, idx)
    s.build(k)
    info = s.info()
    s.close()
    s = gridlib.Scene(0)
    s.set_geometry(verts, idx)
    s.reserve(info["ncells"], info["nrefs"])
    return s


def test_no_spheres_where_no_build_writes_them(gridlib):
    """A crowded scene of more ids than the cluster sort's bitmap span, and a
    batch's sizing builds: one build each, none for spheres."""
    rng = np.random.default_rng(8)
    n = (1 << 20) + 1
    v = rng.uniform(-1, 1, size=(n, 1, 3)) + rng.uniform(-0.004, 0.004, size=(n, 3, 3))
    v[:6000] = rng.uniform(-1e-3, 1e-3, size=(6000, 3, 3)) + np.array([0.3, 0.2, 0.1])
    s = _reserved(gridlib, v.astype(np.float32).reshape(-1, 3), np.arange(3 * n, dtype=np.int32).reshape(-1, 3), 1)
    first, again = _launches(gridlib, lambda: s.build(1)), _launches(gridlib, lambda: s.build(1))
    off, _ = s.download()
    assert np.diff(off).max() > 4096 and first == again
    s.close()

    sc = _crowd("tiny", 9000)
    s = _reserved(gridlib, sc.verts, sc.idx, 1)
    batch = []
    sizing = _launches(gridlib, lambda: batch.append(gridlib.Batch([s], [1], [])))
    own = _launches(gridlib, lambda: s.build(1))          # now with spheres: two builds
    assert 2 * sizing == own
    assert _launches(gridlib, lambda: s.build(1)) == sizing
    batch[0].close()
    s.close()
