"""The ray tracer's specular term at the values where its pow is left out.

Spheres of zero, one-channel and full specular colour with shininess from
negative to 300, lit from the front and from behind (bases from 0 to 1),
against the CPU restatement of the reference (Raytracer::Shade,
muon/integration.cc:74-124). A zero colour times an infinite pow (base 0,
negative shininess) is NaN in both. The tolerance is that of the reference's
films: a few last-place differences of the transcendental, 1e-5 relative plus
1e-6 absolute.
"""
import numpy as np
import pytest

import muon_gb300 as m
from muon_gb300 import native
from oracle import port


def _scene(specular):
    rows = ["film_size 96 64", "camera 0 0 9  0 0 0  0 1 0  45", "integrator raytracer", "max_depth 3",
            "point_light 3 4 6  0.8 0.7 0.6", "point_light 8 1 -4  0.5 0.5 0.7",
            "directional_light 0 0.2 -1  0.4 0.5 0.6", "directional_light 0 -0.1 1  0.3 0.3 0.3",
            "ambient 0.1 0.1 0.1"]
    for k, shine in enumerate((-2, 0, 0.5, 1, 17, 300)):
        rows += ["diffuse 0.2 0.4 0.3", f"specular {specular}", f"shininess {shine}",
                 f"sphere {-3 + 3 * (k % 3)} {1.5 - 3 * (k // 3)} 0 1.2"]
        # a triangle facing away from the camera, towards a light behind it: bases of 0
        x, y = -3 + 3 * (k % 3), 2.9 - 2.9 * (k // 3)
        rows += ["start_mesh", f"vertex {x - 0.8} {y - 0.4} -2", f"vertex {x} {y + 0.4} -2",
                 f"vertex {x + 0.8} {y - 0.4} -2", "tri 0 1 2", "end_mesh"]
    return "\n".join(rows) + "\n"


@pytest.mark.gpu
@pytest.mark.parametrize("specular", ["0 0 0", "0 0.6 0", "0.5 0.4 0.3"])
def test_specular_term_matches_the_oracle(lib, specular):
    text = _scene(specular)
    ref = port.render(text, spp=1, threads=1).film32.reshape(64, 96, 3)
    got = m.Scene.from_string(text).render(pixel_samples=1, intersect_mode=native.ISECT_EXACT).sum.astype(np.float32)
    assert np.array_equal(np.isnan(got), np.isnan(ref))
    assert np.array_equal(np.isinf(got), np.isinf(ref))
    fin = np.isfinite(ref)
    assert np.isnan(ref).any() or np.isinf(ref).any()  # the infinite pow is reached
    assert fin.mean() > 0.5 and (ref[fin] > 0.2).any()
    assert np.all(np.abs(got[fin] - ref[fin]) <= 1e-5 * np.abs(ref[fin]) + 1e-6)
