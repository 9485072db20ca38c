"""Surfaces that overlap within rounding: where a hit's computed distance lies before its leaf's box, which of two
surfaces a ray hits depends on the order its walk meets them in.  That order is the tree's alone: the image is
the same bit for bit whatever the shape of the launch.
"""
import numpy as np
import pytest

import rustracer_gb300 as rt

from test_gpu_traverse import CAM, lit, width  # noqa: F401

pytestmark = pytest.mark.gpu


def offset_layers(layers, n=24):
    """Coplanar layers of tiles, a few rounding errors apart and shifted against each other, so that the tiles a
    ray meets are in different records."""
    rng = np.random.default_rng(5)
    s = rt.Scene()
    mats = [s.add_material(rt.lambertian(c)) for c in ((0.9, 0.2, 0.2), (0.2, 0.9, 0.2), (0.3, 0.3, 0.9))]
    w = 4.2 / n
    for layer in range(layers):
        x0, y0 = -2.1 + rng.uniform(0, w, 2)
        for i in range(-1, n):
            for j in range(-1, n):
                x, y = x0 + w * i, y0 + w * j
                z = np.float32(-0.37) - np.float32(rng.integers(0, 3)) * np.float32(2.0 ** -24)
                s.add_mesh([[x, y, z], [x + w, y, z], [x + w, y + w, z], [x, y + w, z]], [0, 1, 2, 0, 2, 3],
                           mats[layer % 3])
    return lit(s)


def slivers(n, thin, gap):
    """n needles of width `thin` in planes a little behind a tiled wall: their computed distances are off by far
    more than rounding, some to before the wall."""
    rng = np.random.default_rng(3)
    s = rt.Scene()
    wall, needle = (s.add_material(rt.lambertian(c)) for c in ((0.9, 0.2, 0.2), (0.2, 0.9, 0.2)))
    xs, ys = np.linspace(-2.5, 2.5, 13), np.linspace(-2.0, 2.0, 13)
    for x, x1 in zip(xs, xs[1:]):
        for y, y1 in zip(ys, ys[1:]):
            s.add_mesh([[x, y, 0], [x1, y, 0], [x1, y1, 0], [x, y1, 0]], [0, 1, 2, 0, 2, 3], wall)
    centre, along, angle = rng.uniform((-1.5, -1.8), (1.5, 1.8), (n, 2)), rng.uniform(0.5, 2.0, n), rng.uniform(0.3, 1.2, n)
    u, v = along[:, None] * np.stack([-np.ones(n), np.ones(n), rng.uniform(-1, 1, n)], 1), thin * rng.uniform(-1, 1, (n, 3))
    c, d = np.cos(angle)[:, None], np.sin(angle)[:, None]
    p = np.stack([centre[:, :1] + c * u - d * v, centre[:, 1:] + d * u + c * v,
                  np.repeat(-gap * rng.uniform(0.5, 3.0, (n, 1)), 3, axis=1)], axis=-1)
    s.add_mesh(p.reshape(-1, 3), np.arange(3 * n), needle)
    return lit(s)


SCENES = {"two layers": lambda: offset_layers(2), "six layers": lambda: offset_layers(6),
          "slivers 1e-2": lambda: slivers(8000, 1e-2, 1e-5), "slivers 1e-4": lambda: slivers(8000, 1e-4, 1e-3)}


@pytest.fixture(scope="module", params=list(SCENES))
def overlapping(request, gpu):
    return SCENES[request.param]()


def image(scene, w=601, h=403, **tuning):
    r = rt.Renderer(scene, rt.RenderConfig(width=w, height=h, spp=1, accumulate_frames=1, enable_denoise=False,
                                           max_bounces=2))
    r.update_camera(CAM)
    r.tuning = dict(r.tuning, **tuning)
    r.record_frame()
    out = r.read_accumulation()
    r.close()
    return out


def test_which_lane_walks_a_ray_does_not_matter(overlapping, width):  # noqa: F811
    ref = image(overlapping, steps=1)
    for tuning in (dict(block_threads=64), dict(block_threads=256, chunk=64), dict(refill_idle=12)):
        assert np.array_equal(image(overlapping, steps=1, **tuning), ref), tuning
