"""The two variants of the traversal kernels over one tree: a scene of at least
8,192 nodes takes the one that leaves the descent early, a batch of that one
scene the full descent."""
import numpy as np
import pytest

import muon_gb300 as m
from muon_gb300 import native, scenes

DEEP = {
    "mesh": lambda: scenes.dense_mesh(160, 120, 4, 6, 5, 3000, 2),
    "slit_room": lambda: scenes.slit_room(160, 120, 4, 6, 6, 5000, 1),
}


@pytest.fixture(scope="module", params=sorted(DEEP))
def deep(request):
    scene = m.Scene.from_string(DEEP[request.param]())
    assert scene.bvh()[0]["nodes"] >= 8192
    yield scene
    scene.close()


@pytest.mark.gpu
@pytest.mark.parametrize("mode", [native.ISECT_EXACT, native.ISECT_FAST])
@pytest.mark.parametrize("depth", [1, 6])
def test_both_variants_find_the_same_hits(lib, deep, mode, depth):
    """To the bit, in every pixel: the same tree, so that a wrong or missed hit
    of either variant shows, and no surfaces of these scenes that cameras see
    coincide."""
    params = deep.params(intersect_mode=mode, max_depth=depth, seed=3)
    film = deep.render(params)
    batch = m.Batch([deep])
    full = batch.render([params])[0]
    batch.close()
    assert np.array_equal(film.sum, full.sum) and np.array_equal(film.sum_sq, full.sum_sq)
    assert np.array_equal(film.count, full.count)
    assert (film.sum > 0).any(axis=-1).mean() > 0.1  # (the slit room is dark)


@pytest.mark.gpu
@pytest.mark.parametrize("mode", [native.ISECT_EXACT, native.ISECT_FAST, native.ISECT_WATERTIGHT])
@pytest.mark.parametrize("depth,rr", [(6, 0), (-1, 1)])
def test_deep_walks_do_not_depend_on_their_neighbours(lib, deep, mode, depth, rr):
    """Rays are handed to lanes as these become free, and a queue of fewer rays
    than the grid has lanes is spread over all warps: films rendered again and
    in other wavefronts (4 x 19,200 rays at once, one to sixteen a warp) are the
    same bits."""
    kw = dict(intersect_mode=mode, max_depth=depth, russian_roulette=rr, seed=3)
    film = deep.render(**kw)
    for wave_paths in (0, 2 * 19200, 10007, 4864, 0):
        other = deep.render(wave_paths=wave_paths, **kw)
        assert np.array_equal(film.sum, other.sum) and np.array_equal(film.count, other.count)


@pytest.mark.gpu
def test_counters_are_those_of_the_walk_that_renders(lib):
    """Lanes that hold a leaf test boxes in vain while the others descend, more
    of them in the full descent: shadow rays of this scene test 21% more boxes
    so (repeated renders differ by 0.1%). A batch, which takes the full descent
    without counters, has to count that one."""
    scene = m.Scene.from_string(DEEP["slit_room"]())
    params = scene.params(seed=3, flags=native.RENDER_STATS)
    scene.render(params)
    early = scene.stats()
    batch = m.Batch([scene])
    batch.render([params])
    full = batch.stats()[0]
    batch.close()
    scene.close()
    assert full["occlude_rays"] == early["occlude_rays"] > 100000
    assert full["occlude_box_tests"] > 1.1 * early["occlude_box_tests"]
    assert full["extend_box_tests"] > 1.005 * early["extend_box_tests"]
    assert full["occlude_prim_tests"] == early["occlude_prim_tests"]


@pytest.mark.gpu
def test_previews_take_the_full_descent(lib):
    """Camera rays walk together, and leaving their descent early made previews
    of deep trees slower. The counters tell the variants apart: over the same
    rays the full descent tests 1.3% more boxes on this tree."""
    scene = m.Scene.from_string(scenes.dense_mesh(160, 120, 4, 6, 6, 5000, 1))
    assert scene.bvh()[0]["nodes"] >= 8192
    kw = dict(seed=3, flags=native.RENDER_STATS)
    scene.render(max_depth=1, **kw)
    early = scene.stats()
    for integrator in ("normals", "albedo", "depth"):
        scene.render(integrator=integrator, **kw)
        full = scene.stats()
        assert full["extend_rays"] == early["extend_rays"] == 160 * 120 * 4
        assert full["extend_box_tests"] > 1.005 * early["extend_box_tests"]
    scene.close()
