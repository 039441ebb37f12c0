"""Lists above 4,096 entries are tested by bounding spheres first: with thin,
large and coincident triangles in the crowded cells, and rays from
near and far, every hit and occlusion is that of testing every entry, bit for
bit."""
import numpy as np
import pytest

from gridrt import scenes

pytestmark = pytest.mark.gpu


def _crowd(kind, n):
    """n triangles crowded into one corner of a box of 60 others."""
    rng = np.random.default_rng(len(kind))
    c = rng.uniform(-0.02, 0.02, size=(n, 1, 3))
    off = rng.uniform(-1, 1, size=(n, 3, 3))
    if kind == "thin":
        off *= rng.choice([1.0, 1e-3, 1e-5], size=(n, 1, 3)) * 0.01
    elif kind == "mixed":
        off *= np.where(np.arange(n) % 17 == 0, 0.5, 0.002).reshape(-1, 1, 1)
    else:
        off *= 0.002
    v = c + off
    if kind == "twice":
        v[n // 2:] = v[:n - n // 2]          # equal distances: the smaller id wins
    box = rng.uniform(-4, 4, size=(60, 1, 3)) + rng.uniform(-0.3, 0.3, size=(60, 3, 3))
    v = np.concatenate([box, v]).astype(np.float32)
    a = np.cross((v[:, 1] - v[:, 0]).astype(np.float64), (v[:, 2] - v[:, 0]).astype(np.float64))
    v = v[np.sqrt((a * a).sum(1)) > 1e-12]
    return scenes.Scene(verts=v.reshape(-1, 3), idx=np.arange(3 * len(v), dtype=np.int32).reshape(-1, 3))


@pytest.mark.parametrize("kind", ["tiny", "thin", "mixed", "twice"])
@pytest.mark.parametrize("n", [9000, 40000])
def test_crowded_lists(gridlib, kind, n):
    sc = _crowd(kind, n)
    s = gridlib.Scene(0)
    s.set_geometry(sc.verts, sc.idx)
    s.build(1)
    off, _ = s.download()
    assert np.diff(off).max() > 4096
    mid = sc.verts.reshape(-1, 3, 3)[60:].mean(axis=(0, 1))
    rng = np.random.default_rng(n)
    rays = scenes.random_rays(rng, 6000, mid - 4, mid + 4)
    rays[:5000, 4:7] = (mid + rng.normal(size=(5000, 3)) * 0.01 - rays[:5000, 0:3]).astype(np.float32)
    rays[:1000, 0:3] -= 40 * rays[:1000, 4:7]                     # from far outside the box
    rays[5000:, 0:3] = mid + rng.normal(size=(1000, 3)) * 0.01    # from inside the crowd
    seg = rays.copy()
    seg[:, 7] = rng.uniform(0.2, 1.2, size=len(seg))
    s.set_tuning(heavy_cell=0, lanes=2)      # the group walk: every entry tested and decided exactly
    want = s.trace_nearest(rays).view(np.int32), s.trace_any(seg)
    for records in (False, True):
        for lanes in (4, 2):
            s.set_tuning(heavy_cell=32, lanes=lanes, cell_records=records)
            s.build(1)
            for _ in range(2):
                assert np.array_equal(s.trace_nearest(rays).view(np.int32), want[0]), (kind, records, lanes)
                assert np.array_equal(s.trace_any(seg), want[1]), (kind, records, lanes)
                s.build_async(1)
    s.close()
