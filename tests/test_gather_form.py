"""Which form of the gather pass a frame takes: the launches that bench.py counts, on the CPU, and on a GPU the
kernels a profiler sees, at both limits of the one-launch form for the SMs that are there.
"""
import pytest

import bench
import rustracer_gb300 as rt


def config(w, h, **kw):
    return rt.RenderConfig(**{**dict(width=w, height=h, spp=1, max_bounces=4, enable_denoise=False), **kw})


def room():
    return rt.Scene.icosphere_room(level=3, seed=2, sigma=0.02, tex_size=32)


def test_counted_launches(lib):
    cornell, rooms = rt.Scene.cornell555(), room()
    assert bench.wide_records(cornell) <= 64 < bench.wide_records(rooms)
    per_stage = 2 + 2 * 4 + 2 + 1  # four iterations, none of them with a try for the last paths; and the resolve
    assert bench.frame_launches([(cornell, config(256, 256))], 152) == 2
    assert bench.frame_launches([(cornell, config(256, 256, enable_denoise=True))], 152) == 4
    assert bench.frame_launches([(cornell, config(304, 409))], 152) == 2
    assert bench.frame_launches([(cornell, config(304, 410))], 152) == per_stage
    assert bench.frame_launches([(rooms, config(304, 256))], 152) == 2
    assert bench.frame_launches([(rooms, config(304, 257))], 152) == per_stage
    assert bench.frame_launches([(rooms, config(304, 128)), (rooms, config(304, 129))], 152) == per_stage + 1
    assert bench.frame_launches([(rooms, config(1920, 1080, spp=4, max_bounces=8))], 152) == 2 + 2 * 32 + 9 + 2 + 1


def kernels(renderer):
    """The renderer's kernels in one frame (none: there is no profiler here)."""
    torch = pytest.importorskip("torch")
    from torch.profiler import ProfilerActivity, profile

    torch.zeros(1, device="cuda")
    for _ in range(3):  # (the first sessions of a process may see nothing)
        with profile(activities=[ProfilerActivity.CUDA]) as p:
            renderer.record_frame()
            renderer.synchronize()
            torch.cuda.synchronize()
        names = [(e.key, e.count) for e in p.key_averages() if "rtd::" in e.key]
        if names:
            return names
    return []


@pytest.mark.gpu
@pytest.mark.parametrize("name", ["cornell", "room"])
@pytest.mark.parametrize("past", [0, 1])
def test_forms_at_the_limits(gpu, name, past):
    torch = pytest.importorskip("torch")
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    scene = rt.Scene.cornell555() if name == "cornell" else room()
    limit = 512 * sms
    if name == "cornell":
        limit += limit // 5 * 3
    cfg = config(sms, limit // sms + past)  # (a row beyond the limit)
    r = rt.Renderer(scene, cfg)
    r.update_camera(scene.default_camera())
    seen = kernels(r)
    r.close()
    if not seen:
        pytest.skip("no kernel profiler on this machine")
    assert any("wf_paths_kernel" in k for k, _ in seen) == (past == 0)
    assert sum(n for _, n in seen) == bench.frame_launches([(scene, cfg)], sms)


@pytest.mark.gpu
def test_last_paths_in_one_launch(gpu):
    """A larger frame tries for its last paths before every third shade, and a profiled one never."""
    from rustracer_gb300 import _abi as A

    scene = room()
    cfg = config(420, 300, spp=4, max_bounces=6)
    r = rt.Renderer(scene, cfg)
    r.update_camera(scene.default_camera())
    seen = kernels(r)
    if not seen:
        pytest.skip("no kernel profiler on this machine")
    assert sum(n for k, n in seen if "wf_paths_kernel" in k) == 7
    r.set_profiling(A.PROFILE_EVENTS)
    assert not any("wf_paths_kernel" in k for k, _ in kernels(r))
    r.close()
