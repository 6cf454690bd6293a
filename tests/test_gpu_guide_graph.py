"""Frame graphs of one guide and the guides that come after it."""
import numpy as np
import pytest

import muon_gb300 as m
from muon_gb300 import native, scenes


def _frames(scene, guide, film, n):
    """n frames with the same settings (the second is captured, the others replay
    it), then the samples that the pool has seen, and training on them."""
    import torch

    for _ in range(n):
        guide.render_device(scene.params(seed=3, max_depth=4), *[x.data_ptr() for x in film])
    torch.cuda.synchronize()
    guide.train(1)
    return [x.cpu().numpy() for x in film] + [guide.samples(), guide.params()]


@pytest.mark.gpu
def test_a_guide_does_not_replay_the_graph_of_a_destroyed_one(lib):
    """A captured frame holds the addresses of all of its guide's arrays. The
    next guide of the scene has some at the same addresses and others not, by
    what else was freed in between; each of these has to render, fill its pool
    and train as the same guide does for a scene that never had another."""
    import torch

    text = scenes.slit_room(64, 48, 8, 4, level=3, clutter=200, seed=4)
    scene = m.Scene.from_string(text)
    film = [torch.zeros((48, 64, 3), dtype=torch.float64, device="cuda"),
            torch.zeros((48, 64, 3), dtype=torch.float64, device="cuda"),
            torch.zeros((48, 64), dtype=torch.int32, device="cuda")]
    # (a bounce has at most two samples a path, 49,152: none overwrites another of its own)
    configs = [dict(pool_capacity=1 << 17), dict(pool_capacity=1 << 16), dict(pool_capacity=50000),
               dict(pool_capacity=1 << 17, mixture_fraction=0.8), dict(pool_capacity=1 << 16, batch=1 << 11)]
    configs = [dict(dict(seed=2, batch=1 << 12, wave_paths=1 << 16), **c) for c in configs]
    alone = []
    for c in configs:
        fresh = m.Scene.from_string(text)
        guide = m.Guide(fresh, **c)
        alone.append(_frames(fresh, guide, film, 3))
        guide.close()
        fresh.close()
    held = []
    for turn in range(3):
        for k, c in enumerate(configs):
            guide = m.Guide(scene, **c)
            got = _frames(scene, guide, film, 3)
            for a, b in zip(got, alone[k]):
                assert np.array_equal(a, b)
            guide.forward(np.zeros((100 + 1000 * turn, 8), dtype=np.float32))
            guide.close()
            # small blocks come and go between two guides
            held.append(m.Guide(scene, batch=64, wave_paths=256, pool_capacity=64, targets=native.GUIDE_ALL))
            if (turn + k) % 2:
                held.pop(0).close()
    for guide in held:
        guide.close()
    scene.close()
