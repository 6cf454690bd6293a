"""A scene and a batch after a call that the device's memory did not allow."""
import numpy as np
import pytest

import muon_gb300 as m
from muon_gb300 import scenes


@pytest.mark.gpu
def test_a_scene_renders_on_after_a_failed_allocation(lib):
    """Wavefronts of one path of unbounded depth: 20 million of them want 338 GB
    of queue counters in one block, which no device gives. The arrays that the
    scene had before, and a captured frame's graph, may be gone by then; the
    next frames have to find new ones, and no error that is not theirs."""
    text = scenes.cornell(64, 64, 4, 5, 1)
    scene, other = m.Scene.from_string(text), m.Scene.from_string(text)
    frames = [dict(seed=3), dict(seed=3, max_depth=-1, russian_roulette=1), dict(seed=3, wave_paths=5000)]
    want = [other.render(**kw) for kw in frames]
    other.close()
    for kw in frames:
        for _ in range(3):  # captured, then replayed
            scene.render(**kw)
        with pytest.raises(m.MuonError) as e:
            scene.render(pixel_samples=5000, wave_paths=1, max_depth=-1, seed=3)
        assert "out of memory" in str(e.value)
        for again, film in zip(frames, want):
            for _ in range(3):
                got = scene.render(**again)
                assert np.array_equal(got.sum, film.sum) and np.array_equal(got.count, film.count)
    scene.close()
