"""What Scene.intersect and Scene.occluded hand to the library, without a GPU:
the arrays behind the pointers of a call that records them instead."""
import ctypes as C

import numpy as np
import pytest

import muon_gb300 as m


class Recorder:
    """Stands in for the library: keeps copies of a query's input arrays."""

    def _floats(self, pointer, count):
        return np.ctypeslib.as_array((C.c_float * count).from_address(pointer)).copy()

    def muon_gpu_intersect_arrays(self, scene, origins, directions, n, mode, *results):
        self.o, self.d = (self._floats(p, 3 * n).reshape(n, 3) for p in (origins, directions))
        return 0

    def muon_gpu_occluded_arrays(self, scene, origins, directions, limits, n, mode, result):
        self.o, self.d = (self._floats(p, 3 * n).reshape(n, 3) for p in (origins, directions))
        self.limits = self._floats(limits, n)
        return 0


@pytest.fixture
def recorded(monkeypatch):
    recorder, scene = Recorder(), m.Scene.__new__(m.Scene)
    scene._h = None
    monkeypatch.setattr(m, "load", lambda: recorder)
    return scene, recorder


def forms(v):
    """An (n, 3) array in the forms that an assignment to one takes."""
    wide = np.zeros((len(v), 7))
    wide[:, 2:5] = v
    return [v, v.tolist(), v.astype(np.float64), np.asfortranarray(v), wide[:, 2:5], v.astype(">f4"),
            v[None], v[None, None].astype(np.float64)]


@pytest.mark.parametrize("n", [1, 5])
def test_vectors_convert_like_an_assignment(recorded, n):
    """Every form that `rays[:, :3] = vectors` takes, leading axes of length 1
    and one vector for all rays among them; what it refuses is refused."""
    scene, recorder = recorded
    rng = np.random.default_rng(n)
    o, d = rng.normal(size=(2, n, 3)).astype(np.float32)
    for k, dd in enumerate(forms(d) + [d[0], d[:1], d[0].tolist(), d[:1][None]]):
        want = np.zeros((n, 6), dtype=np.float32)
        want[:, :3], want[:, 3:] = forms(o)[k % 6], dd
        for call in (lambda oo: scene.intersect(oo, dd), lambda oo: scene.occluded(oo, dd, np.ones(n))):
            call(forms(o)[k % 6])
            assert np.array_equal(recorder.o, want[:, :3]) and np.array_equal(recorder.d, want[:, 3:])
    for bad in (np.zeros((n + 1, 3)), np.zeros((n, 2)), np.zeros((2, n, 3)), np.zeros((3, n + 1))):
        with pytest.raises(ValueError):
            scene.intersect(o, bad)
        with pytest.raises(ValueError):
            scene.occluded(o, bad, np.ones(n))


@pytest.mark.parametrize("n", [2, 5])
def test_limits_hold_a_value_for_every_ray(recorded, n):
    """Fewer limits than rays were read past their end; one limit serves all
    rays, and of more than n values the first n count, as before."""
    scene, recorder = recorded
    rng = np.random.default_rng(n)
    o, d = rng.normal(size=(2, n, 3)).astype(np.float32)
    for short in (np.ones(n - 1), np.ones(0), []):
        if np.size(short) != 1:
            with pytest.raises(ValueError):
                scene.occluded(o, d, short)
    for one in (1.5, np.float32(1.5), [1.5], np.full((1, 1), 1.5)):
        scene.occluded(o, d, one)
        assert np.array_equal(recorder.limits, np.full(n, 1.5, dtype=np.float32))
    far = rng.uniform(0, 2, 2 * n).astype(np.float32)
    for many in (far[:n], far[:n, None], far[:n].tolist(), far[:n].astype(np.float64), far, far.reshape(2, n)):
        scene.occluded(o, d, many)
        assert np.array_equal(recorder.limits, far[:n])
    scene.occluded(o, d, far[::2])
    assert np.array_equal(recorder.limits, far[::2])
    assert scene.occluded(np.zeros((0, 3)), np.zeros((0, 3)), []).shape == (0,)
