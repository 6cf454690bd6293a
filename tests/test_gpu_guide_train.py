"""The training step's kernels at the edges of their tiles, against the FP64
oracle."""
import numpy as np
import pytest

import muon_gb300 as m
from muon_gb300 import scenes
from oracle import guiding as G


@pytest.mark.gpu
@pytest.mark.parametrize("n", [1, 7, 31, 33, 127, 128, 129, 4097, 304 * 64, 304 * 64 + 1])
def test_gradients_at_tile_edges(lib, n):
    """Batches around the tiles of the layer products (128 samples), the
    loss (32) and the chunks of the weight gradients (64 samples until 304
    chunks are full, then 96). FP32 sums of n products err by about
    sqrt(n) units in the last place of the largest, 1e-5 at most here; ten times
    that."""
    scene = m.Scene.from_string(scenes.cornell(8, 8, 1, 2, 1))
    guide = m.Guide(scene, seed=3, batch=1 << 12, wave_paths=1 << 12, pool_capacity=1 << 12)
    rng = np.random.default_rng(n)
    feat = rng.uniform(0, 1, (n, 8)).astype(np.float32)
    d = rng.normal(size=(n, 3))
    d = (d / np.linalg.norm(d, axis=1, keepdims=True)).astype(np.float32)
    w = rng.uniform(0, 2, n).astype(np.float32)
    grad, loss = guide.gradients(feat, d, w)
    params = G.unflatten(guide.params())
    out, acts, zs = G.forward(params, feat.astype(np.float64), bf16_round=False)
    ref_loss, dout = G.loss_grad(out, d.astype(np.float64), w.astype(np.float64))
    ref = G.flatten(G.backward(params, acts, zs, dout)).astype(np.float64)
    assert abs(loss - ref_loss) <= 1e-5 * max(abs(ref_loss), 1e-3)
    assert np.abs(grad - ref).max() <= 1e-4 * np.abs(ref).max()
    again, _ = guide.gradients(feat, d, w)
    assert np.array_equal(again, grad)
    guide.close()
    scene.close()
