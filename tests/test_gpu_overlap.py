"""Work that runs beside other work, to the bit: guided frames against their
serial form, and the scenes of a batch against batches of one."""
import numpy as np
import pytest

import muon_gb300 as m
from muon_gb300 import native, scenes


@pytest.mark.gpu
@pytest.mark.parametrize("targets", [native.GUIDE_DIRECT, native.GUIDE_ALL], ids=["direct", "all"])
@pytest.mark.parametrize("depth", [1, 2, 6])
def test_guided_frames_equal_their_serial_form(lib, targets, depth):
    """The next bounce's rays are traced beside a guided bounce's shadow rays,
    fold and append of training samples; per-kernel timing runs the kernels one
    after another. The same film and number of samples, also when the frame is
    replayed, and, where samples enter the pool in a fixed order (light samples
    alone: the others are appended as their warps come), after training on them
    the same network."""
    import torch

    scene = m.Scene.from_string(scenes.slit_room(96, 64, 8, 5, level=3, clutter=200, seed=4))
    film = [torch.zeros((scene.height, scene.width, 3), dtype=torch.float64, device="cuda"),
            torch.zeros((scene.height, scene.width, 3), dtype=torch.float64, device="cuda"),
            torch.zeros((scene.height, scene.width), dtype=torch.int32, device="cuda")]
    runs = []
    for flags in (native.RENDER_TIMING, 0):
        guide = m.Guide(scene, seed=8, batch=1 << 12, targets=targets)
        run = []
        for _ in range(4):
            guide.render_device(scene.params(seed=60, max_depth=depth, flags=flags), *[x.data_ptr() for x in film])
            torch.cuda.synchronize()
            run += [guide.samples()] + [x.cpu().numpy() for x in film]
        if targets == native.GUIDE_DIRECT:
            guide.train(2)
            run.append(guide.params())
        runs.append(run)
        guide.close()
    scene.close()
    assert all(np.array_equal(a, b) for a, b in zip(*runs))
    assert runs[0][0] > 0 and (runs[0][1] > 0).mean() > 0.2


@pytest.mark.gpu
@pytest.mark.parametrize("flags", [0, native.RENDER_NO_GRAPH], ids=["graph", "launches"])
def test_batched_scenes_equal_batches_of_one(lib, flags):
    """The next bounce's rays of a batch are traced beside a bounce's shadow rays
    and fold. A batch of one scene runs the same kernels over other queues, so
    that other work lies side by side: the same films, and the same again."""
    made = [m.Scene.from_string(t) for t in (
        scenes.cornell(96, 64, 16, 5, 3), scenes.feature_mix(61, 47, 8, "pathtracer", "mis", 6),
        scenes.batch_scene(0, 7, max_tris=20000, resolutions=(96,), spp_range=(4, 8), depth_range=(3, 6)),
        scenes.batch_scene(1, 7, max_tris=20000, resolutions=(64,), spp_range=(4, 8), depth_range=(3, 6)))]
    params = [s.params(seed=5 + i, flags=flags) for i, s in enumerate(made)]
    alone = []
    for s, p in zip(made, params):
        one = m.Batch([s])
        alone.append(one.render([p])[0])
        one.close()
    batch = m.Batch(made)
    for _ in range(4):
        for film, want in zip(batch.render(params), alone):
            assert np.array_equal(film.sum, want.sum) and np.array_equal(film.sum_sq, want.sum_sq)
            assert np.array_equal(film.count, want.count)
    batch.close()
    for s in made:
        s.close()
