"""Surfaces that overlap within rounding: where a hit's computed distance lies before its leaf's box, which of two
surfaces a ray hits depends on the order its walk meets them in.  That order is the tree's alone: the image is
the same bit for bit whatever the shape of the launch.
"""
import ctypes as C
from pathlib import Path

import numpy as np
import pytest

import rustracer_gb300 as rt
from rustracer_gb300 import _abi as A

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


def test_the_rays_of_a_warp_do_not_matter(overlapping, width):  # noqa: F811
    """How often a warp takes new rays, and solo frames against batches and the one-launch form."""
    ref = image(overlapping)
    for tuning in (dict(), dict(steps=1), dict(steps=7, chunk=64), dict(steps=64), dict(block_threads=64, blocks_per_sm=2),
                   dict(block_threads=256, blocks_per_sm=1, chunk=256)):
        assert np.array_equal(image(overlapping, **tuning), ref), tuning
    small = image(overlapping, 201, 133)
    cfg = rt.RenderConfig(width=201, height=133, spp=1, accumulate_frames=1, enable_denoise=False, max_bounces=2)
    rs = [rt.Renderer(overlapping, cfg) for _ in range(5)]
    for r in rs:
        r.update_camera(CAM)
    rs[0].set_profiling(A.PROFILE_EVENTS)
    rs[0].record_frame()
    b = rt.Batch(rs[1:], use_graphs=False)
    b.render_frame()
    for r in rs:
        assert np.array_equal(r.read_accumulation(), small)
    b.close()


def deep_scene(live, passed):
    """A chain of `passed` + `live` nodes towards -z, each with a side subtree that a ray along -z enters, nearer
    ones deeper, so that all of them wait on the stack.  Only the last side's quad (green) lies on the ray, and a red
    one at 200, a leaf of the root.  The `passed` sides lie behind that: a walk that knows its hit leaves them out."""
    s = rt.Scene()
    red, green = s.add_material(rt.emissive((1, 0, 0), 1.0)), s.add_material(rt.emissive((0, 1, 0), 1.0))
    boxes = []

    def tri(z, x, m):
        s.add_mesh([[x - 1, -1, z], [x + 1, -1, z], [x, 1.5, z]], [0, 1, 2], m)
        boxes.append(((x - 1, -1, z), (x + 1, 1.5, z)))

    tri(-200.0, 0.0, red)
    dist = [300.0 - i for i in range(passed)] + [190.0 - 2 * i for i in range(live)]
    for d in dist:
        tri(-d, -40.0, green)
        tri(-d, 0.0 if d == dist[-1] else 40.0, green)
    tri(-30.0, -40.0, green)
    tri(-30.0, 40.0, green)
    nodes = []

    def leaf(p):
        nodes.append((boxes[p][0], boxes[p][1], p, 0, 1))
        return len(nodes) - 1

    def inner(left, right):
        nodes.append((np.minimum(nodes[left][0], nodes[right][0]), np.maximum(nodes[left][1], nodes[right][1]), left,
                      right, 0))
        return len(nodes) - 1

    nodes.append(None)  # the root
    below = inner(leaf(len(boxes) - 2), leaf(len(boxes) - 1))
    for k in reversed(range(len(dist))):
        below = inner(inner(leaf(1 + 2 * k), leaf(2 + 2 * k)), below)
    inner(leaf(0), below)
    nodes[0] = nodes.pop()
    arr = np.zeros(len(nodes), A.np_dtype(A.BVHNode))
    for n, (lo, hi, left, right, count) in zip(arr, nodes):
        n["bbox_min"], n["bbox_max"], n["left_first"], n["right_child"], n["prim_count"] = lo, hi, left, right, count
    prims = np.arange(len(boxes), dtype=np.uint32)
    desc = A.SceneDesc.from_buffer_copy(s.describe())
    desc.bvh_nodes, desc.bvh_node_count = C.cast(arr.ctypes.data, C.POINTER(A.BVHNode)), len(arr)
    desc.bvh_prims, desc.bvh_prim_count = C.cast(prims.ctypes.data, C.POINTER(C.c_uint32)), len(prims)
    desc.keep = (s, arr, prims)
    return desc


@pytest.mark.parametrize("steps", [1, 3, 64])
@pytest.mark.parametrize("live,passed", [(61, 2), (62, 2), (63, 40), (63, 0)])
def test_full_stack(gpu, live, passed, steps):
    """Two-wide records drop what goes beyond 63 waiting entries: boxes behind a hit the walk has met are none."""
    rt.set_traversal_width(2)
    try:
        r = rt.Renderer(deep_scene(live, passed), rt.RenderConfig(width=1, height=1, spp=1, max_bounces=1,
                                                                   accumulate_frames=1, enable_denoise=False))
    finally:
        rt.set_traversal_width(4)
    r.update_camera(rt.Camera((0, 0, 0), (0, 0, -1), (0, 1, 0), 0.01))
    r.tuning = dict(r.tuning, steps=steps)
    r.record_frame()
    red, green, _ = r.read_accumulation().reshape(-1)[:3]
    assert green > red


def cut_out_scene(thin, scale):
    """A floor under a point light, a cut-out leaf, and slivers whose boxes begin a little beyond the light."""
    n = 4000
    rng = np.random.default_rng(2)
    s = rt.Scene()
    tex = np.full((1, 8, 8, 4), 255, np.uint8)
    tex[0, ::2, ::2, 3] = 0
    s.set_textures(A.TEX_ALBEDO, tex)
    floor, needle = s.add_material(rt.lambertian((0.8, 0.8, 0.8))), s.add_material(rt.lambertian((0.2, 0.9, 0.2)))
    leaf = s.add_material(rt.material(A.MAT_LAMBERTIAN, (0.5, 0.9, 0.4), alpha_cutout=True, tex_albedo=0))
    quad = np.array([[-3, -3, 0], [3, -3, 0], [3, 3, 0], [-3, 3, 0]], np.float32)
    s.add_mesh(quad * scale, [0, 1, 2, 0, 2, 3], floor)
    s.add_mesh((0.1 * quad + np.float32([2, 2, 0.2])) * scale, [0, 1, 2, 0, 2, 3], leaf, uvs=[[0, 0], [1, 0], [1, 1], [0, 1]])
    a, along = rng.uniform(0, np.pi, (n, 1)), rng.uniform(0.2, 1.0, (n, 1))
    u, v = along * np.concatenate([-np.ones((n, 1)), np.ones((n, 1)), rng.uniform(-1, 1, (n, 1))], 1), thin * rng.uniform(-1, 1, (n, 3))
    c = rng.uniform(-0.01, 0.01, (n, 2))
    p = np.stack([c[:, :1] + np.cos(a) * u - np.sin(a) * v, c[:, 1:] + np.sin(a) * u + np.cos(a) * v,
                  np.repeat(0.5 + rng.uniform(0.25e-3, 1e-3, (n, 1)), 3, axis=1)], axis=-1)
    s.add_mesh((p * scale).reshape(-1, 3), np.arange(3 * n), needle)
    s.add_light(rt.point_light((0.0, 0.0, 0.5 * scale), (1, 1, 1), 20.0 * scale * scale))
    return s


def cut_out_lit(thin, scale):
    """The pixels whose light is visible."""
    r = rt.Renderer(cut_out_scene(thin, scale), rt.RenderConfig(width=150, height=150, spp=1, accumulate_frames=1,
                                                                enable_denoise=False, max_bounces=1))
    r.update_camera(rt.Camera((0, 0, 4.0 * scale), (0, 0, 0), (0, 1, 0), 60.0))
    r.record_frame()
    return r.read_accumulation()[..., 0] > 0.03


@pytest.mark.parametrize("thin", [1e-3, 1e-5])
@pytest.mark.parametrize("scale", [1.0, 100.0])
def test_slivers_behind_a_light_with_cut_outs(gpu, width, thin, scale):  # noqa: F811
    """With cut-out materials in the scene a light is hidden by the closest hit before it: also by a sliver whose
    box begins beyond the light.  Compared with the pixels that were lit when occlusion rays had no limit and leaves
    no queue (commit 8f6a6e2)."""
    packed = np.load(Path(__file__).parent / "golden" / "cut_slivers.npz")[f"{width}_{thin:g}_{scale:g}"]
    assert np.array_equal(np.packbits(cut_out_lit(thin, scale)), packed)
