"""The bound on a wavefront's memory."""
import pytest

import muon_gb300 as m
from muon_gb300 import scenes


@pytest.mark.gpu
@pytest.mark.parametrize("batched", [False, True], ids=["frame", "batch"])
def test_wavefront_arrays_stay_within_8_gib(lib, batched):
    """A wavefront holds per path 208 bytes (two sets of hits and links among
    them) and 36 per shadow slot. With 65 slots and 824 samples a pixel, 8 GiB
    hold 4,091 pixels of the 4,096: two wavefronts. (One too many fits where
    one of the two sets is not counted.)"""
    spp, slots = 824, 65
    scene = m.Scene.from_string(scenes.cornell(64, 64, spp, 1, 1))
    params = scene.params(light_samples=slots - 1, light_stratify=0, seed=3)
    most = (8 << 30) // (208 + 36 * slots) // spp
    assert most < 64 * 64 <= (8 << 30) // (208 - 12 + 36 * slots) // spp
    if batched:
        batch = m.Batch([scene])
        batch.render([params])
        stats = batch.stats()[0]
        batch.close()
    else:
        scene.render(params)
        stats = scene.stats()
    scene.close()
    assert stats["primary_rays"] == 64 * 64 * spp
    assert stats["shadow_rays"] > 0.2 * 64 * 64 * spp * slots  # (so many slots there are)
    assert stats["extend_launches"] == 2
