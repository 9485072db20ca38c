"""Photon-map lookups where the grid's neighbour cells may be passed over, against the oracle on the same
photons: photons below the grid (kept in its first cells), beyond it (in the cells of the next row or plane),
without a position, on grids of one to many cells, with both radius rules.  Tolerance as in
test_gpu_parity.py.
"""
import numpy as np
import pytest

import rustracer_gb300 as rt

from test_gpu_parity import FRAC, match_frac, oracle_for

pytestmark = pytest.mark.gpu


def photons(n, gp, rng):
    ph = np.zeros(n, rt._abi.np_dtype(rt._abi.Photon))
    lo = np.array([gp.room_min_x, gp.room_min_y, gp.room_min_z], np.float32)
    span = np.array([gp.grid_x, gp.grid_y, gp.grid_z], np.float32) * np.float32(gp.cell_size)
    pos = lo + rng.uniform(-0.2, 1.6, (n, 3)).astype(np.float32) * span
    wall = rng.integers(0, 3, n)  # half of them on the walls of the scene's bounds, both sides
    on = rng.random(n) < 0.5
    at = np.where(rng.random(n) < 0.5, lo[wall] + np.float32(0.5 * gp.cell_size), np.float32(555.0))
    pos[on, wall[on]] = at[on]
    pos[rng.random(n) < 0.01] = np.nan
    ph["position"] = pos
    ph["power"] = rng.random((n, 3), np.float32) * np.float32(30.0) + np.float32(0.01)
    ph["incident"] = rng.normal(size=(n, 3)).astype(np.float32)
    ph["normal"] = rng.normal(size=(n, 3)).astype(np.float32)
    return ph


@pytest.mark.parametrize("profiled", [False, True])  # one launch, or a launch per stage
@pytest.mark.parametrize("grid_max_dim,radius_mode,count", [(3, 1, 300), (4, 1, 300), (5, 1, 2000), (9, 0, 500),
                                                            (9, 1, 4000), (26, 1, 20000), (60, 1, 60000)])
def test_lookups_pass_over_far_cells(gpu, orc, grid_max_dim, radius_mode, count, profiled):
    scene = rt.Scene.cornell555()
    cfg = rt.RenderConfig(width=60, height=44, spp=2, accumulate_frames=1, enable_denoise=False, enable_photon_map=True,
                          photon_count=count, photon_scale=2000.0, grid_max_dim=grid_max_dim,
                          photon_radius_mode=radius_mode)
    cam = scene.default_camera()
    r = rt.Renderer(scene, cfg)
    r.update_camera(cam)
    ph = photons(r.photon_slots(), r.grid_params(), np.random.default_rng(grid_max_dim))
    r.load_photons(ph)
    if profiled:
        r.set_profiling(rt._abi.PROFILE_EVENTS)
    r.record_frame()
    o = oracle_for(orc, scene, cfg, cam)
    o.load_photons(ph)
    o.record_frame()
    assert match_frac(r.read_accumulation(), o.accum) >= FRAC
