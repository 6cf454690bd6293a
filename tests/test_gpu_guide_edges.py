"""Training samples on both sides of every tile and chunk edge."""
import numpy as np
import pytest

import muon_gb300 as m
from muon_gb300 import scenes
from oracle import guiding as G


def chunk(n):
    """Samples per partial sum of the weight gradients: a multiple of 32, at
    least 64, and at most 304 chunks."""
    return (max(-(-n // 304), 64) + 31) // 32 * 32


@pytest.mark.gpu
@pytest.mark.parametrize("n", [129, 4097, 304 * 64, 304 * 64 + 1, 65537, 100000])
def test_gradients_of_the_samples_at_edges(lib, n):
    """Only the samples beside edges (tiles of 128, chunks, the loss's 32, the
    last) have a weight, some 20 of them, so that one lost or taken twice is
    several per cent of every layer's gradient. Sums of so few FP32 products,
    each through five layers of up to 256 terms, err by about 1e-5 of the
    layer's largest; ten times that."""
    scene = m.Scene.from_string(scenes.cornell(8, 8, 1, 2, 1))
    guide = m.Guide(scene, seed=3, batch=1 << 12, wave_paths=1 << 12, pool_capacity=1 << 12)
    rng = np.random.default_rng(n)
    feat = rng.uniform(0, 1, (n, 8)).astype(np.float32)
    d = rng.normal(size=(n, 3))
    d = (d / np.linalg.norm(d, axis=1, keepdims=True)).astype(np.float32)
    edges = {0, 32, 128, n // 128 * 128, chunk(n), 2 * chunk(n), n // 2 // chunk(n) * chunk(n), n // chunk(n) * chunk(n), n}
    at = sorted({i for e in edges for i in (e - 1, e) if 0 <= i < n})
    w = np.zeros(n, dtype=np.float32)
    w[at] = rng.uniform(0.5, 2, len(at)) * n / len(at)
    grad, loss = guide.gradients(feat, d, w)
    params = G.unflatten(guide.params())
    guide.close()
    scene.close()
    # samples of weight zero add nothing: the gradient of the others, over n
    out, acts, zs = G.forward(params, feat[at].astype(np.float64), bf16_round=False)
    ref_loss, dout = G.loss_grad(out, d[at].astype(np.float64), w[at].astype(np.float64))
    scale = len(at) / n
    ref = G.backward(params, acts, zs, dout * scale)
    assert abs(loss - ref_loss * scale) <= 1e-5 * abs(ref_loss * scale)
    for (gw, gb), (rw, rb) in zip(G.unflatten(grad), ref):
        for got, want in ((gw, rw), (gb, rb)):
            assert np.abs(got - want).max() <= 1e-4 * np.abs(want).max()
