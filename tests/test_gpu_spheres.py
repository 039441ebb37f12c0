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
