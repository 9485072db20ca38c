"""The work a user of rustracer_gb300 has it do, as timed cases.

listed() holds the fixed cases, draw() gives more of the same ranges, prepare() builds what a
program holds before the call (scene, renderer, read-back buffers in pinned memory) from a case and
a seed, run() is one pass through the public entry points, work() what a pass cannot do without,
exact() the 64-bit value of a pass's outputs where there is one.

Kinds of case:

  frames  a renderer: camera in, `frames` progressive frames, the picture read back (the rgba8 image
          the app shows, or the float accumulation the headless entry saves).  With photons the map
          is built beforehand; with `relight` the lights change and the map is rebuilt in the pass.
  batch   one progressive frame of several renderers at once (rt_batch_*), every accumulation read.
  serve   a burst of requests to the request loop (rt_server_*), rendered to their budgets.
  grid    the photon grid of device-resident photons (rt_stage_photon_grid_noalloc).
  post    the denoise and resolve stages on a host renderer's buffers (stage_denoise, stage_resolve).
"""
from __future__ import annotations

import ctypes as C
import math

import numpy as np
import torch

import rustracer_gb300 as rt
from rustracer_gb300 import _abi as A


def listed() -> list[dict]:
    return [
        # The smallest interactive call: one 1 spp frame of the Cornell box while the user orbits the
        # camera, shown at once.  Latency and launches count.
        frames_case("preview_256", scene="cornell", width=256, height=256, spp=1, depth=5, read="rgba8"),
        # The plain method's small workload: 16 progressive frames at 256 x 256, then the raw dump.
        frames_case("headless_256x16", scene="cornell", width=256, height=256, spp=1, depth=5, accumulate=16,
                    frames=16),
        # The app with its default settings (800 x 600, 1 spp, denoise on) in a 20k-triangle room.
        frames_case("app_800x600", scene="room", level=5, tex=256, width=800, height=600, denoise=True),
        # An odd window size, a 328k-triangle room, 3 spp.
        frames_case("room_1003x701", scene="room", level=7, tex=512, width=1003, height=701, spp=3, depth=7,
                    accumulate=32, read="rgba8"),
        # The plain method's large workload and the benchmark's default: 1.31M triangles, 1080p, 4 spp,
        # depth 8.
        frames_case("room_1080p", scene="room", level=8, tex=1024, width=1920, height=1080, spp=4, depth=8,
                    accumulate=32),
        # Cut-out foliage under a sky and a sun: occlusion rays must look at the texture's alpha.
        frames_case("foliage_640x480", scene="foliage", cards=1500, width=640, height=480, spp=2, depth=6,
                    accumulate=32),
        # The photon-map workload after a light change: 2^20 photons traced and binned into 128^3 cells,
        # then a 1080p frame that gathers from them and is denoised.
        frames_case("relight_1080p", scene="cornell", width=1920, height=1080, spp=4, depth=6, accumulate=64,
                    denoise=True, photons=1 << 20, grid=130, radius_mode=1, photon_scale=2000.0, relight=True),
        # The headless entry's photon settings (50,000 photons, the reference's 26-cell grid) while the
        # map stays: four frames of a small room.
        frames_case("photon_view_640x360", scene="room", level=4, tex=128, width=640, height=360, accumulate=4,
                    photons=50_000, frames=4),
        # Many jobs at once: twelve renderers on three resident rooms, mixed sizes, spp, depths, photon
        # maps and denoise.
        {"name": "batch_12", "kind": "batch", "jobs": 12, "level": 5, "rooms": 3},
        # Eight requests arriving together at the request loop, budgets of 2 to 5 frames.
        {"name": "serve_8", "kind": "serve", "jobs": 8, "level": 4, "rooms": 2},
        # A host program's own photons binned on the device, close to the most the entry point takes.
        {"name": "grid_1m", "kind": "grid", "slots": 1_000_003, "dim": 64},
        # A host renderer's noisy frame denoised and tonemapped through host buffers.
        {"name": "post_640x360", "kind": "post", "width": 640, "height": 360},
    ]


def frames_case(name: str | None, *, scene: str, width: int, height: int, level: int = 0, tex: int = 0, cards: int = 0,
                spp: int = 1, depth: int = 0, accumulate: int = 0, denoise: bool = False, photons: int = 0,
                grid: int = 0, radius_mode: int = 0, photon_scale: float = 0.02, relight: bool = False,
                frames: int = 1, read: str = "accumulation") -> dict:
    c = dict(kind="frames", scene=scene, width=width, height=height, level=level, tex=tex, cards=cards, spp=spp,
             depth=depth, accumulate=accumulate, denoise=denoise, photons=photons, grid=grid, radius_mode=radius_mode,
             photon_scale=photon_scale, relight=relight, frames=frames, read=read)
    return c if name is None else {"name": name, **c}


def _log_int(rng, lo: int, hi: int) -> int:
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng) -> dict:
    kind = rng.choice(["cornell", "room", "room", "room", "foliage", "relight", "view", "batch", "serve", "grid", "post"])
    if kind == "batch":
        return {"kind": "batch", "jobs": rng.randint(4, 16), "level": rng.randint(4, 6), "rooms": rng.randint(1, 4)}
    if kind == "serve":
        return {"kind": "serve", "jobs": rng.randint(2, 12), "level": rng.randint(3, 5), "rooms": rng.randint(1, 3)}
    if kind == "grid":
        return {"kind": "grid", "slots": _log_int(rng, 5000, A.NOALLOC_MAX_SLOTS), "dim": rng.randint(8, 64)}
    if kind == "post":
        return {"kind": "post", "width": _log_int(rng, 64, 1920), "height": _log_int(rng, 48, 1080)}
    width, height = _log_int(rng, 48, 1920), _log_int(rng, 40, 1080)
    spp = rng.choice([1, 1, 2, 3, 4])
    depth = rng.randint(3, 8)
    common = dict(width=width, height=height, spp=spp, depth=depth, accumulate=rng.choice([0, 8, 32]),
                  denoise=rng.random() < 0.5)
    if not common["denoise"]:
        common["read"] = rng.choice(["rgba8", "accumulation"])
    if kind == "cornell":
        return frames_case(None, scene="cornell", frames=rng.randint(1, 8), **common)
    if kind == "foliage":
        return frames_case(None, scene="foliage", cards=_log_int(rng, 20, 4000), **common)
    if kind == "relight":
        cells = rng.choice([0, 40, 66, 130])
        return frames_case(None, scene="cornell", photons=_log_int(rng, 4000, 1 << 20), grid=cells,
                           radius_mode=0 if cells == 0 else 1, photon_scale=2000.0, relight=True, **common)
    if kind == "view":
        return frames_case(None, scene="room", level=rng.randint(3, 6), tex=rng.choice([64, 200, 256]),
                           photons=_log_int(rng, 4000, 200_000), frames=rng.randint(1, 4), **common)
    return frames_case(None, scene="room", level=rng.randint(2, 8), tex=rng.choice([64, 300, 512, 1024]), **common)


# ---- scenes ----------------------------------------------------------------------------------------
def foliage(cards: int, rng: np.random.Generator):
    """A ground plane under sky and sun with `cards` leaf cards (two triangles each) whose albedo texture
    is cut out, a few metal and glass panes among them."""
    s = rt.Scene()
    n = 128
    y, x = np.mgrid[0:n, 0:n].astype(np.float32) / n
    tex = np.empty((2, n, n, 4), np.uint8)
    tex[..., :3] = rng.integers(60, 220, (2, n, n, 3), dtype=np.uint8)
    blob = np.sin(9.0 * x + 2.0 * np.sin(7.0 * y)) * np.cos(8.0 * y + 1.5 * np.sin(5.0 * x))
    tex[0, ..., 3] = np.where(blob > -0.2, 255, 0)
    tex[1, ..., 3] = 255
    s.set_textures(A.TEX_ALBEDO, tex)
    ground = s.add_material(rt.material(A.MAT_LAMBERTIAN, (0.8, 0.8, 0.8), roughness=1.0, tex_albedo=1))
    leaf = s.add_material(rt.material(A.MAT_LAMBERTIAN, (0.5, 0.9, 0.4), roughness=1.0, alpha_cutout=True,
                                      tex_albedo=0))
    gold = s.add_material(rt.metal((0.95, 0.64, 0.54), 0.25))
    glass = s.add_material(rt.dielectric(1.5))
    s.add_mesh([[-8, 0, -8], [8, 0, -8], [8, 0, 8], [-8, 0, 8]], [0, 2, 1, 0, 3, 2], ground,
               uvs=[[0, 0], [6, 0], [6, 6], [0, 6]])

    def panes(count: int, material: int, size: float) -> None:
        centre = rng.uniform((-6, 0.3, -6), (6, 3.0, 6), (count, 3))
        u = rng.normal(size=(count, 3))
        u /= np.linalg.norm(u, axis=1, keepdims=True)
        v = np.cross(u, rng.normal(size=(count, 3)))
        v /= np.linalg.norm(v, axis=1, keepdims=True)
        half = size * rng.uniform(0.5, 1.0, (count, 1))
        p = np.stack([centre - half * u - half * v, centre + half * u - half * v, centre + half * u + half * v,
                      centre - half * u + half * v], axis=1)
        idx = (4 * np.arange(count)[:, None] + np.array([0, 1, 2, 0, 2, 3])[None]).astype(np.uint32)
        s.add_mesh(p.reshape(-1, 3), idx, material, uvs=np.tile([[0, 0], [1, 0], [1, 1], [0, 1]], (count, 1)))

    panes(cards, leaf, 0.35)
    panes(max(cards // 40, 1), gold, 0.5)
    panes(max(cards // 40, 1), glass, 0.5)
    s.add_light(rt.environment_light(intensity=0.7))
    s.add_light(rt.directional_light((0.35, 1.0, 0.25), (1.0, 0.95, 0.85), 2.5))
    s.add_light(rt.point_light((0.0, 4.0, 3.0), (1.0, 0.9, 0.8), 6.0))
    return s, rt.Camera((0.0, 2.2, 9.0), (0.0, 1.2, 0.0), (0, 1, 0), 50.0)


def make_scene(case: dict, seed: int, rng: np.random.Generator):
    """(scene, camera): the geometry, materials and view a seed gives."""
    if case["scene"] == "foliage":
        scene, cam = foliage(case["cards"], rng)
    elif case["scene"] == "room":
        scene = rt.Scene.icosphere_room(case["level"], seed % (1 << 31), 0.02, case["tex"])
        cam = scene.default_camera()
    else:
        scene = rt.Scene.cornell555()
        cam = scene.default_camera()
    cam.orbit(float(rng.uniform(-0.15, 0.15)), float(rng.uniform(-0.08, 0.08)))
    return scene, cam


def config_of(c: dict) -> rt.RenderConfig:
    return rt.RenderConfig(width=c["width"], height=c["height"], spp=c["spp"], max_bounces=c["depth"],
                           accumulate_frames=c["accumulate"], enable_denoise=c["denoise"],
                           enable_photon_map=c["photons"] > 0, photon_count=max(c["photons"], 1),
                           photon_scale=c["photon_scale"], grid_max_dim=c["grid"],
                           photon_radius_mode=c["radius_mode"])


def job_config(j: int) -> rt.RenderConfig:
    """The j-th job of a batch or burst: the same mix of sizes and settings for every seed."""
    w, h = [(256, 256), (512, 512), (640, 480), (333, 217)][j % 4]
    photons = [0, 40_000, 0, 0, 150_000][j % 5]
    return rt.RenderConfig(width=w, height=h, spp=[1, 2, 4][j % 3], max_bounces=5 + j % 4, accumulate_frames=0,
                           enable_denoise=j % 4 != 3, enable_photon_map=photons > 0, photon_count=max(photons, 1))


# ---- what a program holds, and one pass --------------------------------------------------------------
def pinned(shape, dtype=torch.float32) -> torch.Tensor:
    return torch.zeros(shape, dtype=dtype, pin_memory=True)


def read_accumulation(r: rt.Renderer, out: torch.Tensor) -> torch.Tensor:
    A.check("rt_read_accumulation", A.load().rt_read_accumulation(r.handle, out.data_ptr(), out.numel()))
    return out


def prepare(case: dict, seed: int) -> dict:
    rng = np.random.default_rng(seed)
    return {"frames": prepare_frames, "batch": prepare_batch, "serve": prepare_serve, "grid": prepare_grid,
            "post": prepare_post}[case["kind"]](case, seed, rng)


def prepare_frames(case, seed, rng):
    scene, cam = make_scene(case, seed, rng)
    cfg = config_of(case)
    r = rt.Renderer(scene, cfg)
    r.update_camera(cam)
    lights = None
    if case["photons"]:
        if case["relight"]:
            lights = [A.Light.from_buffer_copy(scene.describe().lights[i]) for i in range(scene.describe().light_count)]
            for l in lights:
                l.color[:] = tuple(float(v) for v in rng.uniform(8.0, 16.0, 3))
            r.update_lights(lights)
        r.rebuild_photons()
    dtype = torch.uint8 if case["read"] == "rgba8" else torch.float32
    return {"case": case, "scene": scene, "renderer": r, "camera": cam, "lights": lights,
            "out": pinned((case["height"], case["width"], 4), dtype)}


def prepare_batch(case, seed, rng):
    rooms = [rt.Scene.icosphere_room(case["level"], (seed + i) % (1 << 31), 0.02, 256) for i in range(case["rooms"])]
    resident = [rt.ResidentScene(s) for s in rooms]
    rs = []
    for j in range(case["jobs"]):
        r = rt.Renderer(resident[j % case["rooms"]], job_config(j))
        cam = rooms[j % case["rooms"]].default_camera()
        cam.orbit(float(rng.uniform(-0.8, 0.8)), float(rng.uniform(-0.3, 0.3)))
        r.update_camera(cam)
        if job_config(j).enable_photon_map:
            r.rebuild_photons()
        rs.append(r)
    return {"case": case, "rooms": rooms, "resident": resident, "batch": rt.Batch(rs, use_graphs=True),
            "out": [pinned((r.height, r.width, 4)) for r in rs]}


def prepare_serve(case, seed, rng):
    srv = rt.Server(mode="batched", graphs=True)
    rooms = [rt.Scene.icosphere_room(case["level"], (seed + i) % (1 << 31), 0.02, 256) for i in range(case["rooms"])]
    requests = []
    for i, s in enumerate(rooms):
        srv.add_scene(i, s)
    for j in range(case["jobs"]):
        cam = rooms[j % case["rooms"]].default_camera()
        cam.orbit(float(rng.uniform(-0.8, 0.8)), float(rng.uniform(-0.3, 0.3)))
        requests.append((j % case["rooms"], job_config(j), cam, 2 + j % 4))
    return {"case": case, "rooms": rooms, "server": srv, "requests": requests}


def photons_of(case: dict, rng: np.random.Generator):
    """Photons of a room: most on its walls, some in a caustic, some slots empty, a few outside the grid."""
    n, dim = case["slots"], case["dim"]
    gp, _ = rt.derive_grid((np.zeros(3), np.full(3, 10.0)), dim, 1, n)
    lo = np.array([gp.room_min_x, gp.room_min_y, gp.room_min_z], np.float32)
    span = np.array([gp.grid_x, gp.grid_y, gp.grid_z], np.float32) * np.float32(gp.cell_size)
    ph = np.zeros((n, 16), np.float32)
    pos = lo + rng.random((n, 3), np.float32) * span * np.float32(1.02)
    wall = rng.integers(0, 3, n)
    pos[np.arange(n), wall] = lo[wall] + np.where(rng.random(n) < 0.5, np.float32(0.001), np.float32(0.98)) * span[wall]
    spot = rng.random(n) < 0.05
    pos[spot] = lo + span * (np.float32(0.5) + np.float32(0.02) * rng.standard_normal((int(spot.sum()), 3), np.float32))
    ph[:, 0:3] = pos
    ph[:, 4:7] = rng.random((n, 3), np.float32) + np.float32(0.01)
    ph[rng.random(n) < 0.4, 4] = 0.0  # slots of photons that ended early
    ph[:, 8:11] = rng.standard_normal((n, 3), np.float32)
    ph[:, 12:15] = rng.standard_normal((n, 3), np.float32)
    return ph, gp


def prepare_grid(case, seed, rng):
    ph, gp = photons_of(case, rng)
    g = A.GridParams.from_buffer_copy(gp)
    g.photon_slots = case["slots"]
    dev = torch.device("cuda")
    return {"case": case, "gp": g, "photons": torch.from_numpy(ph).to(dev),
            "counts": torch.zeros(g.num_cells, dtype=torch.int32, device=dev),
            "meta": torch.zeros((g.num_cells, 2), dtype=torch.int32, device=dev),
            "sorted": torch.zeros((case["slots"], 16), dtype=torch.float32, device=dev)}


def post_inputs(case: dict, rng: np.random.Generator):
    """A noisy 1 spp-like frame of smooth regions with depth and normal edges, its moments and history."""
    h, w = case["height"], case["width"]
    y, x = np.mgrid[0:h, 0:w].astype(np.float32)
    region = (np.floor(x / 40) + np.floor(y / 30)).astype(np.int32) % 5
    depth = (3.0 + region + 0.002 * x).astype(np.float32)
    normals = rng.standard_normal((5, 3)).astype(np.float32)
    normals /= np.linalg.norm(normals, axis=1, keepdims=True)
    base = rng.uniform(0.1, 0.9, (5, 3)).astype(np.float32)[region]
    frame = np.ones((h, w, 4), np.float32)
    frame[..., :3] = base * rng.gamma(2.0, 0.5, (h, w, 1)).astype(np.float32)
    lum = frame[..., :3] @ np.array([0.2126, 0.7152, 0.0722], np.float32)
    moments = np.zeros((h, w, 4), np.float32)
    moments[..., 0] = lum
    moments[..., 1] = lum * lum * rng.uniform(1.05, 1.8, (h, w)).astype(np.float32)
    gbuffer = np.concatenate([normals[region], depth[..., None]], axis=-1).astype(np.float32)
    accum = np.ones((h, w, 4), np.float32)
    accum[..., :3] = base
    return frame, gbuffer, moments, accum


POST_ALPHA, POST_EXPOSURE = 0.25, 1.2


def prepare_post(case, seed, rng):
    frame, gbuffer, moments, accum = post_inputs(case, rng)
    return {"case": case, "frame": frame, "gbuffer": gbuffer, "moments": moments, "accum": accum}


def run(state: dict):
    kind = state["case"]["kind"]
    if kind == "frames":
        case, r = state["case"], state["renderer"]
        r.update_camera(state["camera"])
        if case["relight"]:
            r.update_lights(state["lights"])
            r.rebuild_photons()
        if case["frames"] > 1:
            r.render_frames(case["frames"])
        else:
            r.record_frame()
        if case["read"] == "rgba8":
            r.read_tonemapped(state["out"].numpy())
            return state["out"]
        return read_accumulation(r, state["out"])
    if kind == "batch":
        b = state["batch"]
        b.render_frame()
        return [read_accumulation(r, o) for r, o in zip(b.renderers, state["out"])]
    if kind == "serve":
        srv = state["server"]
        ids = [srv.submit(*q, keep_result=True) for q in state["requests"]]
        srv.wait_idle()
        images = [srv.result(i) for i in ids]
        for i in ids:
            srv.release(i)
        return images
    if kind == "grid":
        ptr = lambda t: C.c_void_p(t.data_ptr())  # noqa: E731
        A.check("rt_stage_photon_grid_noalloc", A.load().rt_stage_photon_grid_noalloc(
            ptr(state["photons"]), C.byref(state["gp"]), ptr(state["counts"]), ptr(state["meta"]), ptr(state["sorted"]),
            C.c_void_p(torch.cuda.current_stream().cuda_stream)))
        return state["counts"], state["meta"], state["sorted"]
    den = rt.stage_denoise(state["frame"], state["gbuffer"], state["moments"], POST_ALPHA, 2)
    accum, image = rt.stage_resolve(den, state["accum"], POST_ALPHA, exposure=POST_EXPOSURE, gbuffer=state["gbuffer"])
    return den, accum, image


# ---- what a pass cannot do without -------------------------------------------------------------------
# A closest-hit or occlusion ray through a wide tree: boxes tested (6 subtractions, 6 products, 8 min /
# max each) and triangles tested (about 60 operations each); shading a hit, 300 operations.
SEGMENTS_PER_SAMPLE = 3.4  # closest-hit rays of one camera sample in the benchmark's room (depth 8)
TRIANGLES = {"cornell": lambda c: 36, "foliage": lambda c: 2 * c["cards"] + 100,
             "room": lambda c: 20 * 4 ** c["level"] + 12}


def gather_work(triangles: float, pixels: float, spp: int, depth: int, frames: int = 1):
    segments = pixels * max(spp, 1) * frames * min(SEGMENTS_PER_SAMPLE, 0.6 * (depth or 6))
    boxes = 8.0 + 2.0 * math.log2(max(triangles, 2))
    flops = segments * (1.85 * (boxes * 20 + 6 * 60) + 300)
    # triangles with their materials and the tree over them, once; per pixel the accumulated picture in
    # and out, the frame, its moments and the first hit
    return triangles * (128 + 64 + 48 + 20) + frames * pixels * (5 * 16), flops


def denoise_work(pixels: float):
    return 2 * 64.0 * pixels, 2 * 25 * 30.0 * pixels


def grid_work(slots: float, cells: float, binned: float):
    return 16.0 * slots + 8.0 * cells + 128.0 * binned, 10.0 * slots


def job_work(cfg: rt.RenderConfig, triangles: float, frames: int = 1, build: bool = False):
    pixels = float(cfg.width * cfg.height)
    b, f = gather_work(triangles, pixels, cfg.spp, cfg.max_bounces, frames)
    if cfg.enable_denoise:
        db, df = denoise_work(pixels)
        b, f = b + frames * db, f + frames * df
    if cfg.enable_photon_map:
        f += frames * pixels * max(cfg.spp, 1) * 300 * 8.0  # up to 384 photons looked at per diffuse bounce
        if build:
            slots = 6.0 * cfg.photon_count
            gb, gf = grid_work(slots, float(min((cfg.grid_max_dim or 26) ** 3, 1 << 22)), slots / 3.5)
            b, f = b + gb, f + gf + 2.5 * cfg.photon_count * 900
    return b + frames * 4 * pixels, f


def work(case: dict) -> dict:
    kind = case["kind"]
    if kind == "frames":
        b, f = job_work(config_of(case), TRIANGLES[case["scene"]](case), case["frames"], case["relight"])
        return {"bytes": b, "flops": f}
    if kind in ("batch", "serve"):
        tris = TRIANGLES["room"](case)
        b = f = 0.0
        for j in range(case["jobs"]):
            jb, jf = job_work(job_config(j), 0.0, 2 + j % 4 if kind == "serve" else 1, kind == "serve")
            b, f = b + jb, f + jf
        return {"bytes": b + case["rooms"] * tris * 260.0, "flops": f}
    if kind == "grid":
        b, f = grid_work(case["slots"], float(case["dim"] ** 3), 0.6 * case["slots"])
        return {"bytes": b, "flops": f}
    pixels = float(case["width"] * case["height"])
    b, f = denoise_work(pixels)
    return {"bytes": b + 52 * pixels, "flops": f + 60 * pixels}


# ---- 64-bit values -----------------------------------------------------------------------------------
def exact(case: dict, seed: int):
    """A path's decisions (which light, which lobe, whether it goes on) hang on 32-bit values, so a frame
    has no 64-bit value; the photon grid and the image stages do."""
    rng = np.random.default_rng(seed)
    if case["kind"] == "grid":
        ph, gp = photons_of(case, rng)
        lo = (gp.room_min_x, gp.room_min_y, gp.room_min_z)
        cell = np.float32(gp.cell_size)
        g = [np.clip((ph[:, a] - np.float32(lo[a])) / cell, 0, 2.0**31).astype(np.int64) for a in range(3)]
        key = g[0] + g[1] * gp.grid_x + g[2] * gp.grid_x * gp.grid_y
        kept = np.flatnonzero((ph[:, 4] > 0) & (key < gp.num_cells))
        order = kept[np.argsort(key[kept], kind="stable")]
        out = np.zeros(ph.shape, np.float64)
        out[: len(order)] = ph[order]
        return None, None, out
    if case["kind"] == "post":
        frame, gbuffer, moments, accum = (a.astype(np.float64) for a in post_inputs(case, rng))
        den = frame
        for step in (1, 2):
            den = denoise_64(den, gbuffer, moments, step)
        hist = accum * (1.0 - POST_ALPHA) + den * POST_ALPHA
        return den, hist, None
    return None


def denoise_64(frame, gbuffer, moments, step: int):
    """One edge-aware a-trous pass (3 x 3 variance window, 5 x 5 B3-spline taps) in 64 bits."""
    h, w, _ = frame.shape
    weight = np.array([0.2126, 0.7152, 0.0722])

    def shifted(a, dy, dx):
        """a at (y + dy, x + dx) and whether that lies inside the image."""
        ys, xs = np.arange(h) + dy, np.arange(w) + dx
        ok = ((ys >= 0) & (ys < h))[:, None] & ((xs >= 0) & (xs < w))[None, :]
        return a[np.clip(ys, 0, h - 1)][:, np.clip(xs, 0, w - 1)], ok

    var = np.maximum(moments[..., 1] - moments[..., 0] ** 2, 0.0)
    acc, cnt = np.zeros((h, w)), np.zeros((h, w))
    for dy in (-1, 0, 1):
        for dx in (-1, 0, 1):
            v, ok = shifted(var, dy, dx)
            acc += np.where(ok, v, 0.0)
            cnt += ok
    var_c = acc / np.maximum(cnt, 1.0) * (POST_ALPHA / max(2.0 - POST_ALPHA, 1e-4))
    denom_l = var_c * 3.0 + 1e-6
    denom_d = 0.05 * np.maximum(gbuffer[..., 3], 1e-4)
    lum = frame[..., :3] @ weight
    b3 = (0.375, 0.25, 0.0625)
    total, out = np.zeros((h, w)), np.zeros((h, w, 3))
    for dy in range(-2, 3):
        for dx in range(-2, 3):
            g, ok = shifted(gbuffer, dy * step, dx * step)
            c, _ = shifted(frame, dy * step, dx * step)
            l, _ = shifted(lum, dy * step, dx * step)
            k = b3[abs(dx)] * b3[abs(dy)] * np.maximum((gbuffer[..., :3] * g[..., :3]).sum(-1), 0.0) ** 12
            k = k * np.exp(-np.abs(gbuffer[..., 3] - g[..., 3]) / denom_d) * np.exp(-((l - lum) ** 2) / denom_l)
            k = np.where(ok, k, 0.0)
            out += c[..., :3] * k[..., None]
            total += k
    res = np.ones_like(frame)
    res[..., :3] = np.where(total[..., None] > 1e-6, out / np.maximum(total, 1e-300)[..., None], frame[..., :3])
    return res
