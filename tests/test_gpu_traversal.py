"""Variants of the traversal kernels against each other: which one runs is
decided by the size of the scene or of the frame, and results must not depend
on it."""
import numpy as np
import pytest

import muon_gb300 as m
from muon_gb300 import native, scenes


@pytest.mark.gpu
@pytest.mark.parametrize("mode", [native.ISECT_EXACT, native.ISECT_FAST, native.ISECT_WATERTIGHT])
@pytest.mark.parametrize("depth,rr", [(1, 0), (5, 0), (-1, 1)])
def test_deep_tree_descent_changes_no_hits(lib, mode, depth, rr):
    """The same primitives under a tree just below the size at which warps
    leave the descent early, and one just above it (leaves of one primitive):
    the same paths. Two primitives at exactly one distance may swap (at most
    0.5% of rays in the hit fixtures, far fewer here), so all but 2% of the
    pixels have to be equal to the bit."""
    parsed = m.parse_string(scenes.dense_mesh(96, 64, 4, 5, level=4, clutter=4000, seed=4))
    films = []
    for leaf, above in ((0, False), (1, True)):
        scene = m.Scene(parsed, max_leaf_size=leaf)
        assert (scene.bvh()[0]["nodes"] >= 8192) == above
        films.append(scene.render(intersect_mode=mode, max_depth=depth, russian_roulette=rr, seed=9))
        scene.close()
    a, b = films
    assert np.array_equal(a.count, b.count)
    assert (a.sum == b.sum).all(axis=-1).mean() >= 0.98


@pytest.mark.gpu
@pytest.mark.parametrize("width,height", [(1, 1), (5, 3), (152, 33), (61, 80)])
@pytest.mark.parametrize("wave_paths", [31, 1000, 4865])
def test_short_queues_trace_the_same_paths(lib, width, height, wave_paths):
    """Queues of one ray to a few rays per warp, and around one ray for each
    warp of a full grid (4,864 on 152 multiprocessors): the film does not
    depend on how a frame is cut into wavefronts."""
    scene = m.Scene.from_string(scenes.feature_mix(width, height, 2, "pathtracer", "mis", 6))
    whole = scene.render(seed=3)
    cut = scene.render(seed=3, wave_paths=min(wave_paths, 2 * width * height))
    assert np.array_equal(whole.sum, cut.sum) and np.array_equal(whole.sum_sq, cut.sum_sq)
    assert np.array_equal(whole.count, cut.count)


@pytest.mark.gpu
@pytest.mark.parametrize("width,height,paths", [(61, 47, 31), (61, 47, 1023), (61, 47, 1024), (61, 47, 1025),
                                                (96, 64, 4096 + 129), (1301, 1010, 1216 * 1024 - 1),
                                                (1301, 1010, 1216 * 1024 + 1), (1301, 1010, 1301 * 1010)])
def test_class_lists_hold_every_hit(lib, width, height, paths):
    """The stable class partition at the edges of its segments (1,024 entries,
    and one segment per block of a full grid, 1,216 on 152 multiprocessors):
    hits missing from a list, or in it twice, would change the film. Wavefronts
    of `paths` paths against wavefronts of another size."""
    scene = m.Scene.from_string(scenes.feature_mix(width, height, 1, "pathtracer", "mis", 3))
    film = scene.render(seed=2, wave_paths=paths)
    other = scene.render(seed=2, wave_paths=700 if width < 100 else 262144)
    assert np.array_equal(film.sum, other.sum) and np.array_equal(film.count, other.count)
    assert (film.sum > 0).mean() > 0.2


@pytest.mark.gpu
@pytest.mark.parametrize("width,height,spp,depth,nee", [(1, 1, 1, 2, "mis"), (33, 31, 3, 1, "mis"), (129, 127, 7, 5, "off"),
                                                        (129, 127, 7, -1, "mis"), (181, 183, 2, -1, "on")])
def test_overlapped_bounces_render_the_same_film(lib, width, height, spp, depth, nee):
    """Bounces whose next rays are traced beside their shadow rays and fold, in
    one wavefront and in two or three at a time, against kernels run one after
    another (a render with per-kernel timing): bit for bit the same film, also
    when the frame is replayed."""
    scene = m.Scene.from_string(scenes.feature_mix(width, height, spp, "pathtracer", "mis", 5))
    kw = dict(seed=6, max_depth=depth, russian_roulette=1 if depth < 0 else 0, next_event_estimation=nee)
    serial = scene.render(flags=native.RENDER_TIMING, **kw)
    paths = width * height * spp
    for wave_paths in (0, (paths + 1) // 2, (paths + 2) // 3):
        for _ in range(3):
            film = scene.render(wave_paths=wave_paths, **kw)
            assert np.array_equal(film.sum, serial.sum) and np.array_equal(film.sum_sq, serial.sum_sq)
            assert np.array_equal(film.count, serial.count)
    assert scene.stats()["paths"] == paths
