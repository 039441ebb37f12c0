"""The settings a scene has before any tuning are among those a tuner tries, and
can be asked for again."""
import json

import numpy as np
import pytest

from gridrt import autotune, scenes


def test_default_settings_are_tried():
    assert autotune.SPACE["lanes"][0] == -1              # by the launch's size, tried first
    assert 8 in autotune.SPACE["refill"]                 # ray arrays


def test_cached_result_of_another_space_is_searched_again(tmp_path, monkeypatch):
    monkeypatch.setattr(autotune, "CACHE", str(tmp_path / "cache.json"))
    old = {"w": {"best": {"lanes": 1}, "all": [{"cfg": {"lanes": 1}, "ms": 1.0}], "when": 0.0}}
    json.dump(old, open(autotune.CACHE, "w"))            # an entry without its space
    best, _ = autotune.search(lambda c: c["lanes"], space={"lanes": (0, 1)}, key="w", reps=1)
    assert best == {"lanes": 0} and autotune.search.last_source == "search"
    best, _ = autotune.search(lambda c: 0.0, space={"lanes": (0, 1)}, key="w", reps=1)
    assert best == {"lanes": 0} and autotune.search.last_source == "cache"
    best, _ = autotune.search(lambda c: -c["lanes"], space={"lanes": (0, 1, 2)}, key="w", reps=1)
    assert best == {"lanes": 2} and autotune.search.last_source == "search"


@pytest.mark.gpu
def test_lanes_by_size_can_be_asked_for_again(gridlib):
    sc = scenes.plane_and_debris(quads=40, debris=3000)
    s = gridlib.Scene(0)
    s.set_geometry(sc.verts, sc.idx)
    s.build(4)
    rays = scenes.random_rays(np.random.default_rng(2), 1000, sc.verts.min(0), sc.verts.max(0))

    def launches():
        before = gridlib.kernel_launches()
        hits = s.trace_nearest(rays).view(np.int32)
        return gridlib.kernel_launches() - before, hits

    unset, want = launches()
    for lanes in (1, -1, 2, -1):
        s.set_tuning(lanes=lanes)
        n, hits = launches()
        assert np.array_equal(hits, want), lanes
        assert (n == unset) == (lanes == -1), lanes      # 32 lanes a ray: no pass behind it
    for lanes in (0, 3, 8, -2):
        with pytest.raises(gridlib.GridRTError):
            s.set_tuning(lanes=lanes)
    s.close()
