"""Frames around the sizes where the one-launch form of the gather pass takes over, which differ for trees of few
records, and its photon lookups with one and several samples per pixel, alone and in a batch: bit for bit as
with a launch per stage (a profiled frame) and as the same frames rendered alone.
"""
import numpy as np
import pytest

import rustracer_gb300 as rt
from rustracer_gb300 import _abi as A

from test_gpu_paths import check, pool  # noqa: F401

pytestmark = pytest.mark.gpu


# 152 SMs hold 77,824 paths: 304 x 256 pixels, 304 x 409.6 for trees of few records
@pytest.mark.parametrize("name,w,h", [("cornell", 304, 409), ("cornell", 304, 410), ("room", 304, 256), ("room", 304, 257)])
def test_around_the_limits(pool, name, w, h):  # noqa: F811
    check(pool, name, width=w, height=h, spp=1, max_bounces=4)


@pytest.mark.parametrize("name", ["cornell", "room"])
@pytest.mark.parametrize("w,h,spp", [(120, 90, 1), (120, 90, 3), (500, 300, 1), (500, 300, 2)])
def test_photon_lookups(pool, name, w, h, spp):  # noqa: F811
    check(pool, name, width=w, height=h, spp=spp, max_bounces=5, enable_photon_map=True, photon_count=20_000,
          photon_scale=2000.0)


@pytest.mark.parametrize("spps", [(1, 1), (1, 3), (2, 3)])
def test_photon_lookups_in_a_batch(pool, spps):  # noqa: F811
    scene = pool["cornell"][0]
    cfgs = [rt.RenderConfig(width=150 + 40 * i, height=101, spp=s, accumulate_frames=4, enable_photon_map=True,
                            photon_count=10_000, photon_scale=2000.0, enable_denoise=False) for i, s in enumerate(spps)]

    def made():
        rs = [rt.Renderer(scene, c) for c in cfgs]
        for r in rs:
            r.update_camera(scene.default_camera())
            r.rebuild_photons()
        return rs

    alone, batch = made(), rt.Batch(made())
    for r in alone:
        r.set_profiling(A.PROFILE_EVENTS)
        r.record_frame()
    batch.render_frame()
    for a, b in zip(alone, batch.renderers):
        assert np.array_equal(a.read_accumulation(), b.read_accumulation())
