"""The traversal kernels where their queues and stacks overflow their usual sizes, against the oracle:
leaves of one to many triangles, stacks deeper than the part kept in shared memory, ray counts around
the 32 rays a warp reads ahead, with both record widths.  Tolerance as in test_gpu_parity.py (equal-t
hits resolve to the lowest prim slot on both sides, so no path may diverge).
"""
import numpy as np
import pytest

import rustracer_gb300 as rt

from test_gpu_parity import FRAC, match_frac, render_both

pytestmark = pytest.mark.gpu


def lit(s):
    s.add_light(rt.environment_light(intensity=0.8))
    s.add_light(rt.point_light((0.5, 2.0, 6.0), (1.0, 0.9, 0.8), 20.0))
    return s


def fan_scene(blades):
    """Per fan, `blades` triangles around one centroid: no split separates them, so each fan is one leaf."""
    s = rt.Scene()
    grey = s.add_material(rt.lambertian((0.7, 0.7, 0.7)))
    gold = s.add_material(rt.metal((0.9, 0.6, 0.4), 0.3))
    for k, (x, y) in enumerate([(-1.0, -0.5), (0.2, 0.4), (1.1, -0.2)]):
        a = 2 * np.pi * np.arange(blades)[:, None] / (3 * blades) + 2 * np.pi * np.arange(3)[None] / 3
        p = np.stack([x + np.cos(a), y + np.sin(a), np.full_like(a, float(k))], axis=-1)
        s.add_mesh(p.reshape(-1, 3), np.arange(3 * blades), gold if k == 1 else grey)
    return lit(s)


def stacked_scene(n):
    """n large triangles behind one another: a ray enters nearly every box, so a near-first walk keeps as
    many records pending as the tree allows."""
    rng = np.random.default_rng(1)
    s = rt.Scene()
    grey = s.add_material(rt.lambertian((0.7, 0.7, 0.7)))
    glass = s.add_material(rt.dielectric(1.4))
    base = np.array([[-2.0, -1.5, 0.0], [2.0, -1.5, 0.0], [0.0, 2.5, 0.0]])
    p = base[None] + rng.uniform(-0.3, 0.3, (n, 1, 3)) * np.array([1.0, 1.0, 0.0])
    p[:, :, 2] -= np.linspace(0.0, 4.0, n)[:, None] + rng.uniform(0, 1e-3, (n, 3))
    s.add_mesh(p[: n // 2].reshape(-1, 3), np.arange(3 * (n // 2)), glass)
    s.add_mesh(p[n // 2:].reshape(-1, 3), np.arange(3 * (n - n // 2)), grey)
    return lit(s)


CAM = rt.Camera((0.0, 0.2, 5.0), (0.0, 0.0, 0.0), (0, 1, 0), 50.0)


@pytest.fixture(params=[2, 4])
def width(request):
    rt.set_traversal_width(request.param)
    yield request.param
    rt.set_traversal_width(4)


@pytest.mark.parametrize("blades", [1, 3, 5, 9, 77])
def test_leaf_sizes(gpu, orc, width, blades):
    s = fan_scene(blades)
    assert s.arrays()["bvh_nodes"]["prim_count"].max() >= min(blades, 4)
    cfg = rt.RenderConfig(width=40, height=32, spp=2, accumulate_frames=2, enable_denoise=False)
    r, o = render_both(orc, s, cfg, 2, cam=CAM)
    assert match_frac(r.read_accumulation(), o.accum) >= FRAC


@pytest.mark.parametrize("n", [300, 12000])
def test_deep_stacks(gpu, orc, width, n):
    cfg = rt.RenderConfig(width=24, height=20, spp=2, accumulate_frames=1, enable_denoise=False, max_bounces=8)
    r, o = render_both(orc, stacked_scene(n), cfg, 1, cam=CAM)
    assert match_frac(r.read_accumulation(), o.accum) >= FRAC


@pytest.mark.parametrize("w,h", [(1, 1), (31, 1), (32, 1), (33, 1), (127, 3), (613, 7)])
def test_ray_counts(gpu, orc, w, h):
    scene = rt.Scene.cornell555()
    cfg = rt.RenderConfig(width=w, height=h, spp=1, accumulate_frames=1, enable_denoise=False)
    r, o = render_both(orc, scene, cfg, 1)
    assert match_frac(r.read_accumulation(), o.accum) >= FRAC


def layered_scene():
    """Axis-aligned quads in pairs a rounding error apart, tiled edge to edge: a ray's two nearest hits are
    ties or nearly so, and lie no farther than the (flat) boxes they are in."""
    s = rt.Scene()
    mats = [s.add_material(rt.lambertian(c)) for c in ((0.9, 0.2, 0.2), (0.2, 0.9, 0.2), (0.3, 0.3, 0.9))]
    mats.append(s.add_material(rt.metal((0.9, 0.8, 0.5), 0.2)))
    rng = np.random.default_rng(5)
    for layer in range(3):
        for i in range(6):
            for j in range(6):
                x, y = 0.7 * (i - 3), 0.7 * (j - 3)
                z = np.float32(-0.37 - 1.1 * layer) + np.float32(rng.integers(0, 3)) * np.float32(2.0 ** -24)
                quad = [[x, y, z], [x + 0.7, y, z], [x + 0.7, y + 0.7, z], [x, y + 0.7, z]]
                for m in rng.choice(4, 2, replace=False):
                    s.add_mesh(quad, [0, 1, 2, 0, 2, 3], mats[m])
                    quad = [[a, b, c - np.float32(2.0 ** -24)] for a, b, c in quad]
    return lit(s)


def test_near_ties_do_not_depend_on_the_launch(gpu, width):
    """Which rays share a warp, how often it tests leaves and how its jobs are batched change no hit."""
    s = layered_scene()
    cfg = rt.RenderConfig(width=301, height=203, spp=2, accumulate_frames=1, enable_denoise=False, max_bounces=6)

    def image(**tuning):
        r = rt.Renderer(s, cfg)
        r.update_camera(CAM)
        r.tuning = dict(r.tuning, **tuning)
        r.record_frame()
        return r.read_accumulation()

    ref = image()
    for tuning in (dict(), dict(steps=1), dict(steps=7, chunk=64), dict(block_threads=64, blocks_per_sm=2),
                   dict(block_threads=256, blocks_per_sm=1, chunk=256)):
        assert np.array_equal(image(**tuning), ref), tuning
    rs = [rt.Renderer(s, cfg) for _ in range(3)]
    for r in rs:
        r.update_camera(CAM)
    b = rt.Batch(rs, use_graphs=False)
    b.render_frame()
    for r in rs:
        assert np.array_equal(r.read_accumulation(), ref)
    b.close()
