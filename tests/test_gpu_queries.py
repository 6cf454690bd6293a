"""Ray queries: arrays against interleaved records, and queries of different
sizes against each other."""
import ctypes as C

import numpy as np
import pytest

import muon_gb300 as m
from muon_gb300 import native, scenes


def rays_in_box(n, seed):
    rng = np.random.default_rng(seed)
    o = rng.uniform([-0.9, 0.1, -0.9], [0.9, 1.9, 0.9], (n, 3)).astype(np.float32)
    d = rng.normal(size=(n, 3))
    d = (d / np.linalg.norm(d, axis=1, keepdims=True)).astype(np.float32)
    return o, d, rng.uniform(0.1, 2.0, n).astype(np.float32)


@pytest.fixture(scope="module")
def deep():
    scene = m.Scene.from_string(scenes.dense_mesh(16, 16, 1, 2, level=5, clutter=3000, seed=2))
    assert scene.bvh()[0]["nodes"] >= 8192
    yield scene
    scene.close()


@pytest.mark.gpu
@pytest.mark.parametrize("mode", [native.ISECT_EXACT, native.ISECT_FAST, native.ISECT_WATERTIGHT])
@pytest.mark.parametrize("n", [1, 33, 4864, 4865, 8192, 8193, 32 * 4864 - 1, 32 * 4864 + 1, 1 << 19])
def test_queries_of_every_size_agree(lib, deep, mode, n):
    """Around the sizes where the copies (8,192 rays) and the rays per warp change
    (one up to 4,864 rays on 152 multiprocessors, 32 from 32 times that): the
    same answers as a few thousand of the rays asked for alone, also for rays
    inside a box that stands on the floor, and as the interleaved entry points
    give."""
    o, d, far = rays_in_box(n, n)
    dist, prim, pos, nrm = deep.intersect(o, d, mode)
    blocked = deep.occluded(o, d, far, mode)
    assert dist.dtype == np.float32 and prim.dtype == np.int32 and blocked.dtype == bool
    some = np.arange(0, n, max(1, n // 4000))
    pieces = deep.intersect(o[some], d[some], mode)
    for a, b in zip((dist, prim, pos, nrm), pieces):
        assert np.array_equal(a[some], b)
    assert np.array_equal(blocked[some], deep.occluded(o[some], d[some], far[some], mode))
    rays = np.concatenate([o, d], axis=1)
    hits = np.zeros((n, 8), dtype=np.float32)
    out = np.zeros(n, dtype=np.uint8)
    rp = rays.ctypes.data_as(C.POINTER(native.Ray))
    native.check(lib.muon_gpu_intersect(deep._h, rp, n, mode, hits.ctypes.data_as(C.POINTER(native.Hit))))
    native.check(lib.muon_gpu_occluded(deep._h, rp, far.ctypes.data_as(C.POINTER(C.c_float)), n, mode,
                                       out.ctypes.data_as(C.POINTER(C.c_uint8))))
    assert np.array_equal(hits[:, 0], dist) and np.array_equal(hits[:, 1].view(np.int32), prim)
    assert np.array_equal(hits[:, 2:5], pos) and np.array_equal(hits[:, 5:8], nrm)
    assert np.array_equal(out.astype(bool), blocked)
    assert n < 1000 or (0.5 < (prim >= 0).mean() and 0.05 < blocked.mean() < 0.95)


@pytest.mark.gpu
def test_query_inputs_convert_as_before(lib, deep):
    """Lists, float64, strided columns and one direction for all rays."""
    o, d, far = rays_in_box(50, 3)
    want = deep.intersect(o, np.broadcast_to(d[:1], (50, 3)))
    both = np.concatenate([o, d], axis=1)
    for oo, dd in ((o.tolist(), d[0].tolist()), (o.astype(np.float64), d[:1]), (both[:, :3], d[0])):
        for a, b in zip(deep.intersect(oo, dd), want):
            assert np.array_equal(a, b)
        assert np.array_equal(deep.occluded(oo, dd, far), deep.occluded(o, np.broadcast_to(d[:1], (50, 3)), far))
    empty = deep.intersect(np.zeros((0, 3)), np.zeros((0, 3)))
    assert [a.shape for a in empty] == [(0,), (0,), (0, 3), (0, 3)]
    with pytest.raises(ValueError):
        deep.intersect(o, d[:7])
    with pytest.raises(m.MuonError):
        deep.intersect(o, d, 9)
