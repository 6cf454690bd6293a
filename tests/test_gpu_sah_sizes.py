"""The device binned-SAH builder at the sizes where its phases meet.

Subtrees of at most 8 references are built by a lane per reference, nodes up
to 255 by a warp, up to 2,047 by a block, larger ones by chunks of 256 and
more; the counts below lie at these lines, the positions are either even or
spread over five decades (uneven splits: nodes of every size under large
ones). The tree must be the host builder's, node for node and bit for bit.
"""
import numpy as np
import pytest

from test_gpu_sah_build import _same_tree


def _soup(n, spread):
    rng = np.random.default_rng(n)
    c = rng.uniform(-1, 1, (n, 3))
    if spread:
        c *= 10.0 ** rng.uniform(-4, 1, (n, 1))
    v = (c[:, None] + 0.02 * rng.normal(size=(n, 3, 3))).reshape(-1, 3)
    rows = ["film_size 8 8", "camera 0 0 5  0 0 0  0 1 0  45", "start_mesh"]
    rows += ["vertex %.9g %.9g %.9g" % tuple(p) for p in v]
    rows += [f"tri {3 * i} {3 * i + 1} {3 * i + 2}" for i in range(n)]
    return "\n".join(rows + ["end_mesh"]) + "\n"


@pytest.mark.gpu
@pytest.mark.parametrize("spread", [False, True], ids=["even", "spread"])
@pytest.mark.parametrize("n", [2, 7, 8, 9, 31, 33, 255, 256, 257, 2047, 2048, 2049, 5000, 40000, 90001])
def test_device_tree_equals_the_host_tree(lib, n, spread):
    host, dev = _same_tree(_soup(n, spread))
    host.close()
    dev.close()
