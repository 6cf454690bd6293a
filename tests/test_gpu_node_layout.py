"""Nodes in the form that the kernels read, from every builder."""
import numpy as np
import pytest

import muon_gb300 as m

@pytest.mark.gpu
@pytest.mark.parametrize("n", [2, 4096, 4097, 4098])
def test_trees_of_all_builders_find_the_same_hits(lib, n):
    """With one primitive a leaf a tree has n - 1 nodes; the host converts those
    of its own trees up to 4,096 and the device larger ones and all that it
    built. Distances to the bit; the primitives too, but for exact ties."""
    rng = np.random.default_rng(n)
    rows = ["film_size 8 8", "camera 0 0 5  0 0 0  0 1 0  45"]
    rows += ["sphere %.9g %.9g %.9g 0.05" % tuple(c) for c in rng.uniform(-1, 1, (n, 3))]
    parsed = m.parse_string("\n".join(rows) + "\n")
    o = rng.uniform(-1, 1, (20000, 3))
    d = rng.normal(size=(20000, 3))
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    hits = []
    for builder in ("host", "gpu_sah", "gpu"):
        scene = m.Scene(parsed, max_leaf_size=1, builder=builder)
        assert scene.bvh()[0]["nodes"] == n - 1
        hits.append(scene.intersect(o, d)[:2])
        scene.close()
    assert n == 2 or (hits[0][1] >= 0).mean() > 0.2
    for distance, prim in hits[1:]:
        assert np.array_equal(distance, hits[0][0])
        assert (prim == hits[0][1]).mean() >= 0.995
