"""The one-launch form of the gather pass (few pixels, or the last paths of a larger frame) against the
wavefront: a profiled frame runs one launch per stage, so the same frames with and without
profiling must be equal bit for bit, their ray counts too.
"""
import numpy as np
import pytest

import rustracer_gb300 as rt
from rustracer_gb300 import _abi as A

from test_gpu_edge import FEATURE_CAM, feature_scene

pytestmark = pytest.mark.gpu


def scenes():
    return {"cornell": (rt.Scene.cornell555(), None), "feature": (feature_scene(), FEATURE_CAM),
            "room": (rt.Scene.icosphere_room(level=3, seed=2, sigma=0.02, tex_size=32), None),
            "empty": (rt.Scene(), None)}


@pytest.fixture(scope="module")
def pool(gpu):
    return scenes()


def frames(scene, cam, cfg, profiled):
    r = rt.Renderer(scene, cfg)
    r.update_camera(cam or scene.default_camera())
    if cfg.enable_photon_map:
        r.rebuild_photons()
    if profiled:
        r.set_profiling(A.PROFILE_EVENTS)
    r.render_frames(2)
    st = r.stats()
    out = [r.read_accumulation(), r.read_moments(), r.read_gbuffer(), r.read_tonemapped()]
    r.close()
    return out, (st.segments, st.shadow_rays)


def check(pool, name, **kw):
    scene, cam = pool[name]
    cfg = rt.RenderConfig(accumulate_frames=4, enable_denoise=False, **kw)
    one, n_one = frames(scene, cam, cfg, False)
    wave, n_wave = frames(scene, cam, cfg, True)
    assert n_one == n_wave
    for a, b in zip(one, wave):
        assert np.array_equal(a.view(np.uint8), b.view(np.uint8))


@pytest.mark.parametrize("name", ["cornell", "feature", "room", "empty"])
@pytest.mark.parametrize("w,h,spp,depth", [(1, 1, 1, 6), (7, 3, 9, 3), (33, 17, 2, 8), (200, 131, 3, 5)])
def test_whole_frames(pool, name, w, h, spp, depth):
    check(pool, name, width=w, height=h, spp=spp, max_bounces=depth)


@pytest.mark.parametrize("w,h", [(304, 255), (304, 256), (304, 257), (512, 152)])  # 512 pixels per SM: 304 x 256
def test_around_the_limit(pool, w, h):
    check(pool, "feature", width=w, height=h, spp=1, max_bounces=4)


@pytest.mark.parametrize("name", ["cornell", "feature", "room"])
@pytest.mark.parametrize("photons", [False, True])
def test_last_paths_of_a_larger_frame(pool, name, photons):
    check(pool, name, width=420, height=300, spp=4, max_bounces=6, enable_photon_map=photons, photon_count=20000,
          photon_scale=50.0)


@pytest.mark.parametrize("debug", [False, True])
def test_photon_maps(pool, debug):
    check(pool, "room", width=90, height=61, spp=3, max_bounces=6, enable_photon_map=True, photon_count=20000,
          photon_scale=50.0, photon_debug=debug)


def test_batches_of_few_pixels(pool):
    """Several scenes in one launch: each image is its image rendered alone by the wavefront."""
    specs = [("cornell", 64, 48, 2), ("feature", 40, 25, 3), ("room", 31, 17, 1), ("feature", 9, 5, 4)]
    rs = []
    for name, w, h, spp in specs:
        scene, cam = pool[name]
        r = rt.Renderer(scene, rt.RenderConfig(width=w, height=h, spp=spp, accumulate_frames=4, enable_denoise=False))
        r.update_camera(cam or scene.default_camera())
        rs.append(r)
    b = rt.Batch(rs, use_graphs=True)
    b.render_frames(2)
    segments = 0
    for r, (name, w, h, spp) in zip(rs, specs):
        scene, cam = pool[name]
        cfg = rt.RenderConfig(width=w, height=h, spp=spp, accumulate_frames=4, enable_denoise=False)
        wave, n = frames(scene, cam, cfg, True)
        segments += n[0]
        assert np.array_equal(r.read_accumulation(), wave[0]), name
    assert b.stats().segments == segments
    b.close()
