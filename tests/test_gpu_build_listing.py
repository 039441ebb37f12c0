"""The count and scatter passes list a warp's references lane by lane or over
the whole warp, by the triangles' sizes and the scene's: both, and mixtures
inside one scene, give the oracle's grid bit for bit."""
import numpy as np
import pytest

from gridrt import scenes

pytestmark = pytest.mark.gpu


def _soup(rng, n, half):
    c = rng.uniform(-1, 1, size=(n, 1, 3))
    v = (c + rng.uniform(-1, 1, size=(n, 3, 3)) * np.asarray(half).reshape(-1, 1, 1)).astype(np.float32)
    return scenes.Scene(verts=v.reshape(-1, 3), idx=np.arange(3 * n, dtype=np.int32).reshape(n, 3))


@pytest.mark.parametrize("name", ["alike", "one large a warp", "few tiny", "flat rows", "warp edges", "above one wave"])
@pytest.mark.parametrize("k", [1, 6])
def test_listing(gridlib, oracle, name, k):
    import torch
    rng = np.random.default_rng(len(name))
    wave = 2048 * torch.cuda.get_device_properties(0).multi_processor_count
    if name == "alike":
        sc = _soup(rng, 700, np.full(700, 0.2))
    elif name == "one large a warp":
        sc = _soup(rng, 1024, np.where(np.arange(1024) % 32 == 5, 0.5, 0.004))
    elif name == "few tiny":
        sc = _soup(rng, 1024, np.where(np.arange(1024) % 32 < 20, 0.001, 0.12))
    elif name == "flat rows":          # ranges of one cell along y or z
        sc = _soup(rng, 640, np.full(640, 0.1))
        v = sc.verts.reshape(-1, 3, 3)
        v[::2, :, 1] = v[::2, :1, 1]
        v[1::4, :, 2] = v[1::4, :1, 2]
    elif name == "warp edges":
        sc = _soup(rng, 33, np.full(33, 0.3))
    else:
        sc = _soup(rng, wave + 1, np.full(wave + 1, 0.01))
    s = gridlib.Scene(0)
    s.set_geometry(sc.verts, sc.idx)
    s.build(k)
    g = oracle.Grid(sc.verts, sc.idx, k)
    off, ids = s.download()
    assert np.array_equal(off, g.offsets) and np.array_equal(ids, g.ids)
    s.build_async(k)
    assert s.build_check() == 0
    off, ids = s.download()
    assert np.array_equal(off, g.offsets) and np.array_equal(ids, g.ids)


@pytest.mark.parametrize("n", [1, 8, 9, 32, 33, 256, 257, 4096, 4097])
def test_longest_list_of_a_scene(gridlib, oracle, n):
    """A list of as many entries as the scene has triangles, at the sizes where
    the sorts of longer lists are no longer launched."""
    rng = np.random.default_rng(n)
    sc = _soup(rng, n, np.full(n, 0.2))
    v = sc.verts.reshape(-1, 3, 3)
    v[:] = v * 1e-4 + np.float32([0.21, 0.33, -0.27])
    v[rng.integers(n)] = [[0.0, 0.0, 0.0], [1.0, 1.0, 0.5], [-1.0, -0.5, -1.0]]   # its range covers every cell
    s = gridlib.Scene(0)
    s.set_geometry(sc.verts, sc.idx)
    g = oracle.Grid(sc.verts, sc.idx, 2)
    assert np.diff(g.offsets).max() == n
    s.build(2)
    off, ids = s.download()
    assert np.array_equal(off, g.offsets) and np.array_equal(ids, g.ids)
    s.build_async(2)
    assert s.build_check() == 0
    off, ids = s.download()
    assert np.array_equal(off, g.offsets) and np.array_equal(ids, g.ids)
