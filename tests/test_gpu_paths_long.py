"""Paths whose sample or segment number leaves its 16 bits: the one-launch form of the gather pass takes as many
steps as the wavefront has iterations, with the same images and ray counts.
"""
import numpy as np
import pytest

import rustracer_gb300 as rt

from test_gpu_paths import check

pytestmark = pytest.mark.gpu


def mirror_box():
    """A closed box of perfect mirrors around the camera (a dielectric whose Fresnel term rounds to 1): no path ends
    by itself."""
    s = rt.Scene()
    mirror = s.add_material(rt.dielectric(1e9))
    p = np.array([[x, y, z] for x in (-2, 2) for y in (-2, 2) for z in (-2, 2)], np.float32)
    idx = [0, 1, 3, 0, 3, 2, 4, 6, 7, 4, 7, 5, 0, 4, 5, 0, 5, 1, 2, 3, 7, 2, 7, 6, 0, 2, 6, 0, 6, 4, 1, 5, 7, 1, 7, 3]
    s.add_mesh(p, idx, mirror)
    s.add_light(rt.point_light((0.5, 1.0, 0.3), (1.0, 0.9, 0.8), 20.0))
    return s


@pytest.fixture(scope="module")
def scenes(gpu):
    return {"cornell": (rt.Scene.cornell555(), None),
            "mirrors": (mirror_box(), rt.Camera((0.3, 0.1, 1.0), (0.2, 0.3, -1.0), (0, 1, 0), 70.0))}


@pytest.mark.parametrize("spp", [65536, 65537])
def test_samples(scenes, spp):
    check(scenes, "cornell", width=5, height=3, spp=spp, max_bounces=1)


@pytest.mark.parametrize("depth", [300, 65536, 65600])
def test_segments(scenes, depth):
    check(scenes, "mirrors", width=9, height=4, spp=1, max_bounces=depth)
