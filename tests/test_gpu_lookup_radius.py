"""A photon radius set after create, of either sign: only its square enters a lookup, so the sign must not decide which
cells are passed over, least of all on a grid one cell thick whose photons lie beside it (and are kept in the cells
of the next plane).
"""
import dataclasses

import numpy as np
import pytest

import rustracer_gb300 as rt

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("profiled", [False, True])  # one launch, or a launch per stage
@pytest.mark.parametrize("cells", [0.4, 1.05, 1.1, 1.25, 30.0])
def test_sign_of_the_radius(gpu, cells, profiled):
    scene = rt.Scene()
    grey = scene.add_material(rt.lambertian((0.8, 0.8, 0.8)))
    scene.add_mesh([[0, 0, 0], [1, 0, 0], [1, 0, 1], [0, 0, 1]], [0, 2, 1, 0, 3, 2], grey)
    cfg = rt.RenderConfig(width=400, height=400, spp=1, accumulate_frames=1, enable_denoise=False, enable_photon_map=True,
                          photon_count=16, photon_scale=2000.0, grid_max_dim=9, photon_radius_mode=1)
    images = []
    for sign in (1.0, -1.0):
        rng = np.random.default_rng(3)
        r = rt.Renderer(scene, cfg)
        r.update_camera(rt.Camera((0.5, 2.0, 0.5), (0.5, 0.0, 0.5), (0, 0, 1), 30.0))
        gp = r.grid_params()
        assert gp.grid_y == 1
        ph = np.zeros(r.photon_slots(), rt._abi.np_dtype(rt._abi.Photon))
        pos = rng.uniform(0, 1, (len(ph), 3))
        pos[:, 1] = rng.uniform(0.5, 1.2, len(ph)) * gp.cell_size
        ph["position"], ph["power"] = pos, rng.uniform(0.1, 1.0, (len(ph), 3))
        ph["incident"] = [0.0, -1.0, 0.0]
        r.load_photons(ph)
        r.config = dataclasses.replace(r.config, photon_radius=sign * cells * gp.cell_size)
        if profiled:
            r.set_profiling(rt._abi.PROFILE_EVENTS)
        r.record_frame()
        images.append(r.read_accumulation())
    assert np.array_equal(*images)
    assert cells < 0.5 or images[0][..., 0].max() > 0.1  # (0.024 without photons)
