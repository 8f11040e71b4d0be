"""Performance cases: what programs that use this renderer have it do.

Every case goes through the public entry points (the classes of
wgpu_spectral_rt_b200 and, where a program owns the buffers, the C ABI of
include/srt.h).  Sizes are those of bench.py's workloads, the headless
driver's defaults and the tests, or generic ones; `draw` spreads further
cases over the same ranges.

    listed()            the named cases
    draw(rng)           one more case of the same ranges
    prepare(case, seed) scene, renderer and buffers a program holds before the call
    run(state)          one pass
    work(case)          bytes and operations a pass cannot do without
    exact(case, seed)   None: the outputs are images of a Monte-Carlo estimate
                        drawn from 32-bit random streams (no 64-bit value), or
                        whole numbers
"""
from __future__ import annotations

import ctypes as C
import math

import numpy as np
import torch

import wgpu_spectral_rt_b200 as srt

# ---------------------------------------------------------------------------- cases


def listed() -> list[dict]:
    return [
        # one preview frame of the prism scene at thumbnail size (the sizes of the tests): launch latency
        {"name": "prism_thumb_96x64", "kind": "frame", "preset": srt.PRESET_CUSTOM_PRISM, "scene_seed": 0,
         "width": 96, "height": 64, "depth": 12, "photons": 1 << 16, "frames": 1, "restart": False, "guide": "off",
         "read": "ldr"},
        # the headless driver's defaults: the Cornell box at 640 x 480, one frame shown per pass
        {"name": "cornell_640x480", "kind": "frame", "preset": srt.PRESET_CORNELL_BOX, "scene_seed": 0,
         "width": 640, "height": 480, "depth": 12, "photons": 1 << 20, "frames": 1, "restart": False, "guide": "off",
         "read": "ldr"},
        # bench.py's config 1: a small image rendered to 16 spp from a cleared accumulation, read as FP32
        {"name": "config1_256_spp16", "kind": "frame", "preset": srt.PRESET_CONFIG1, "scene_seed": 0,
         "width": 256, "height": 256, "depth": 8, "photons": 1 << 18, "frames": 16, "restart": True, "guide": "off",
         "read": "accum"},
        # bench.py's config 2 (1.57M triangles, 4M photons per frame): the next frame of a progressive render
        {"name": "config2_1080p", "kind": "frame", "preset": srt.PRESET_CONFIG2, "scene_seed": 0,
         "width": 1920, "height": 1080, "depth": 12, "photons": 1 << 22, "frames": 1, "restart": False,
         "guide": "off", "read": "ldr"},
        # the caustic slab at 1080p, depth 16: long paths and a dense photon map
        {"name": "slab_1080p", "kind": "frame", "preset": srt.PRESET_CAUSTIC_SLAB, "scene_seed": 0,
         "width": 1920, "height": 1080, "depth": 16, "photons": 1 << 20, "frames": 1, "restart": False,
         "guide": "off", "read": "ldr"},
        # the same scene with the path guide (a trained network kept fixed: the final render of a guided job)
        {"name": "slab_guided_960x540", "kind": "frame", "preset": srt.PRESET_CAUSTIC_SLAB, "scene_seed": 0,
         "width": 960, "height": 540, "depth": 16, "photons": 1 << 20, "frames": 1, "restart": False,
         "guide": "frozen", "read": "accum"},
        # the indirectly lit room at an odd size, guided, 4 spp from a cleared accumulation
        {"name": "indirect_guided_801x451", "kind": "frame", "preset": srt.PRESET_INDIRECT_ROOM, "scene_seed": 0,
         "width": 801, "height": 451, "depth": 12, "photons": 1 << 18, "frames": 4, "restart": True,
         "guide": "frozen", "read": "accum"},
        # several seeded scenes at once, each with its own viewport and accumulation (data generation)
        {"name": "batch_8_scenes", "kind": "batch", "scenes": 8, "scene_seed": 1, "size_min": 192, "size_max": 512,
         "depth": 12, "photons": 1 << 20, "frames": 2},
        # an animated scene: instances move, the tree is refitted, one frame is rendered and shown
        {"name": "animate_512x384", "kind": "animate", "scene_seed": 3, "moved": 16, "width": 512, "height": 384,
         "depth": 12, "photons": 1 << 19},
        # opening a scene: upload, tree build, a new renderer, the first two frames
        {"name": "open_331k_triangles", "kind": "open", "preset": srt.PRESET_BATCH_RANDOM, "scene_seed": 4,
         "width": 640, "height": 480, "depth": 12, "photons": 1 << 18, "frames": 2},
        # ray queries from a host program against the config-2 geometry, an odd number of them
        {"name": "rays_config2_250007", "kind": "rays", "preset": srt.PRESET_CONFIG2, "scene_seed": 0,
         "rays": 250_007, "any_hit": False},
        # the photon hash grid on buffers the caller owns (no allocation), near its largest photon set
        {"name": "grid_device_1000003", "kind": "grid", "photons": 1_000_003, "hash_bits": 22},
    ]


def _log_int(rng, lo: int, hi: int) -> int:
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng) -> dict:
    kind = rng.choice(["frame"] * 5 + ["batch", "animate", "open", "rays", "grid"])
    if kind == "frame":
        preset = rng.choice([srt.PRESET_CORNELL_BOX, srt.PRESET_CUSTOM_PRISM, srt.PRESET_CONFIG1,
                             srt.PRESET_CAUSTIC_SLAB, srt.PRESET_INDIRECT_ROOM, srt.PRESET_BATCH_RANDOM])
        w = _log_int(rng, 64, 1400)
        h = max(48, int(w * rng.uniform(0.5, 1.0)))
        frames = rng.choice([1, 1, 2, 4]) if w * h < 250_000 else 1
        return {"kind": "frame", "preset": preset, "scene_seed": rng.randint(1, 8), "width": w, "height": h,
                "depth": rng.randint(4, 16), "photons": _log_int(rng, 1 << 14, 1 << 20), "frames": frames,
                "restart": frames > 1, "guide": rng.choice(["off", "off", "frozen"]),
                "read": rng.choice(["ldr", "accum"])}
    if kind == "batch":
        return {"kind": "batch", "scenes": rng.randint(2, 6), "scene_seed": rng.randint(1, 40), "size_min": 64,
                "size_max": rng.randint(96, 384), "depth": rng.randint(6, 14),
                "photons": _log_int(rng, 1 << 16, 1 << 19), "frames": rng.choice([1, 2])}
    if kind == "animate":
        return {"kind": "animate", "scene_seed": rng.choice([2, 3, 4, 8]), "moved": rng.randint(1, 12),
                "width": rng.randint(120, 720), "height": rng.randint(90, 480), "depth": rng.randint(6, 14),
                "photons": _log_int(rng, 1 << 15, 1 << 19)}
    if kind == "open":
        return {"kind": "open", "preset": rng.choice([srt.PRESET_CONFIG1, srt.PRESET_BATCH_RANDOM]),
                "scene_seed": rng.randint(1, 8), "width": rng.randint(120, 720), "height": rng.randint(90, 480),
                "depth": rng.randint(6, 14), "photons": _log_int(rng, 1 << 15, 1 << 18),
                "frames": rng.choice([1, 2])}
    if kind == "rays":
        return {"kind": "rays", "preset": rng.choice([srt.PRESET_CORNELL_BOX, srt.PRESET_BATCH_RANDOM]),
                "scene_seed": rng.randint(1, 8), "rays": _log_int(rng, 500, 300_000),
                "any_hit": rng.random() < 0.4}
    return {"kind": "grid", "photons": _log_int(rng, 300, 1 << 20), "hash_bits": rng.randint(18, 24)}


# ---------------------------------------------------------------------------- state

# Geometry a program has loaded on the host (scene builders of the presets), by (preset, scene seed).
_builders: dict = {}


def _builder(preset: int, scene_seed: int):
    key = (preset, scene_seed)
    if key not in _builders:
        b = srt.SceneBuilder()
        cam = b.add_preset(preset, scene_seed)
        _builders[key] = (b, cam)
    return _builders[key]


def _stream_seed(seed: int) -> int:
    return (seed * 2654435761 + 97) & 0x7FFFFFFF


def _pinned(*shape, dtype):
    return torch.zeros(shape, dtype=dtype, pin_memory=True)


def _ok(status: int, ctx) -> None:
    if status != 0:
        raise srt.SrtError(status, (srt.lib().srt_get_error_string(ctx.h) or b"").decode())


def _read(renderer, buffer) -> torch.Tensor:
    """The image into the caller's pinned buffer: RGBA8 rows or FP32 sums."""
    p = C.c_void_p(buffer.data_ptr())
    if buffer.dtype == torch.uint8:
        _ok(srt.lib().srt_read_ldr_rgba8(renderer.h, p, 4 * renderer.target_width), renderer.ctx)
    else:
        _ok(srt.lib().srt_read_accum_f32(renderer.h, p), renderer.ctx)
    return buffer


def _room_rays(n: int, half: np.ndarray, mid: np.ndarray, seed: int) -> np.ndarray:
    """Rays from points of a room in uniform directions: origin, tmin, direction, tmax."""
    g = np.random.default_rng(seed)
    r = np.empty((n, 8), np.float32)
    r[:, 0:3] = mid + half * g.uniform(-1.0, 1.0, (n, 3))
    r[:, 3] = 1e-4
    d = g.normal(size=(n, 3))
    r[:, 4:7] = d / np.linalg.norm(d, axis=1, keepdims=True)
    r[:, 7] = 100.0
    return r


def prepare(case: dict, seed: int) -> dict:
    kind = case["kind"]
    s: dict = {"case": case, "step": 0}
    if kind == "grid":
        # a caustic on the floor plus photons spread over the room, a few without energy
        n = case["photons"]
        g = torch.Generator(device="cuda").manual_seed(seed)
        pos = torch.rand((n, 3), generator=g, device="cuda") * 2.0 - 1.0
        caustic = torch.rand(n, generator=g, device="cuda") < 0.7
        spot = torch.randn((n, 3), generator=g, device="cuda") * 0.25
        spot[:, 1] = -1.0 + 1e-4 * spot[:, 1]
        pos = torch.where(caustic[:, None], spot, pos)
        wavelength = 380.0 + 400.0 * torch.rand((n, 1), generator=g, device="cuda")
        d = torch.randn((n, 3), generator=g, device="cuda")
        d = d / d.norm(dim=1, keepdim=True)
        energy = torch.rand((n, 1), generator=g, device="cuda")
        energy = torch.where(energy < 0.01, torch.zeros_like(energy), energy)
        s["photons"] = torch.cat([pos, wavelength, d, energy], dim=1).contiguous()
        s["keys"] = torch.zeros(n, dtype=torch.int64, device="cuda")
        s["ranges"] = torch.zeros((1 << case["hash_bits"], 2), dtype=torch.int32, device="cuda")
        s["frame"] = seed % 1000
        return s
    s["ctx"] = ctx = srt.Context(0)
    if kind == "batch":
        g = np.random.default_rng(case["scene_seed"])
        scenes, sizes, params, cams = [], [], [], []
        for k in range(case["scenes"]):
            b, cam = _builder(srt.PRESET_BATCH_RANDOM, case["scene_seed"] + k)
            scenes.append(b.build(ctx))
            sizes.append(tuple(int(x) for x in g.integers(case["size_min"], case["size_max"] + 1, 2)))
            params.append(srt.default_params(max_depth=case["depth"], photons_per_frame=case["photons"],
                                             seed=(_stream_seed(seed) + k) & 0x7FFFFFFF))
            cams.append(srt.CameraController(*cam))
        s["batch"] = srt.Batch(ctx, scenes, sizes, params)
        s["cameras"] = cams
        s["buffers"] = [_pinned(h, w, 4, dtype=torch.float32) for w, h in sizes]
        return s
    preset = srt.PRESET_BATCH_RANDOM if kind == "animate" else case["preset"]
    b, cam = _builder(preset, case["scene_seed"])
    if kind == "open":
        s["builder"], s["camera"] = b, srt.CameraController(*cam)
        s["params"] = srt.default_params(max_depth=case["depth"], photons_per_frame=case["photons"],
                                         seed=_stream_seed(seed))
        s["buffer"] = _pinned(case["height"], case["width"], 4, dtype=torch.uint8)
        return s
    s["scene"] = scene = b.build(ctx)
    if kind == "rays":
        config2 = preset == srt.PRESET_CONFIG2
        half = np.array([3.9, 1.95, 3.9] if config2 else [0.95, 0.95, 0.95])
        s["rays"] = _room_rays(case["rays"], half, np.array([0.0, 1.0 if config2 else 0.0, 0.0]), seed)
        return s
    flags = 0
    if case.get("guide", "off") == "frozen":
        flags = srt.FLAG_GUIDING | srt.FLAG_GUIDE_FROZEN
    w, h = case["width"], case["height"]
    p = srt.default_params(max_depth=case["depth"], photons_per_frame=case["photons"], seed=_stream_seed(seed),
                           flags=flags)
    s["camera"] = srt.CameraController(*cam)
    s["renderer"] = r = srt.Renderer(ctx, scene, w, h, p)
    if flags:
        r.set_guide_weights(srt.guide_default_weights(1 + seed % 1000))
    read = case.get("read", "ldr")
    s["buffer"] = _pinned(h, w, 4, dtype=torch.uint8 if read == "ldr" else torch.float32)
    if kind == "animate":
        # eight poses of the moved spheres (instances 7.. of the seeded scene, column-major object to world): each
        # circles its built place by about its own radius, as an animation moves an object between frames
        g = np.random.default_rng(seed)
        n = case["moved"]
        s["ids"] = np.arange(7, 7 + n, dtype=np.uint32)
        a = b.arrays()
        t = np.array([list(a.instances[int(i)].transform) for i in s["ids"]], np.float32)[None].repeat(8, axis=0)
        angle = 2.0 * math.pi * (np.arange(8)[:, None] / 8.0 + g.uniform(0.0, 1.0, (1, n)))
        t[:, :, 12] += 0.5 * t[:, :, 0] * np.cos(angle)
        t[:, :, 14] += 0.5 * t[:, :, 0] * np.sin(angle)
        s["poses"] = t
    return s


# ---------------------------------------------------------------------------- one pass


def _render(renderer, camera, frames: int) -> None:
    aspect = renderer.target_width / renderer.target_height
    for _ in range(frames):
        renderer.render(camera.build_uniform(aspect, renderer.frame_count))


def run(s: dict):
    case = s["case"]
    kind = case["kind"]
    if kind == "frame":
        r = s["renderer"]
        if case["restart"]:
            r.reset_accumulation()
        _render(r, s["camera"], case["frames"])
        return _read(r, s["buffer"])
    if kind == "batch":
        batch = s["batch"]
        for r in batch.renderers:
            r.reset_accumulation()
        for f in range(case["frames"]):
            batch.render([c.build_uniform(w / h, f) for c, (w, h) in zip(s["cameras"], batch.sizes)])
        return [_read(r, b) for r, b in zip(batch.renderers, s["buffers"])]
    if kind == "animate":
        r = s["renderer"]
        s["scene"].update_instances(s["ids"], s["poses"][s["step"] % 8])
        s["step"] += 1
        r.reset_accumulation()
        _render(r, s["camera"], 1)
        return _read(r, s["buffer"])
    if kind == "open":
        scene = s["builder"].build(s["ctx"])
        r = srt.Renderer(s["ctx"], scene, case["width"], case["height"], s["params"])
        _render(r, s["camera"], case["frames"])
        image = _read(r, s["buffer"])
        r.close()
        scene.close()
        return image
    if kind == "rays":
        hits = s["scene"].trace(s["rays"], any_hit=case["any_hit"])
        if case["any_hit"]:
            return {"prim": hits["prim"]}  # occluded or not: which of the hits was found first is not defined
        return {"t": hits["t"], "prim": hits["prim"], "u": hits["u"], "v": hits["v"]}
    status = srt.lib().srt_photon_grid_build_noalloc(
        C.c_void_p(torch.cuda.current_stream().cuda_stream), C.c_void_p(s["photons"].data_ptr()), case["photons"],
        s["frame"], 0.02, case["hash_bits"], C.c_void_p(s["keys"].data_ptr()), C.c_void_p(s["ranges"].data_ptr()))
    if status != 0:
        raise srt.SrtError(status, "srt_photon_grid_build_noalloc")
    return {"keys": s["keys"], "ranges": s["ranges"]}


# ---------------------------------------------------------------------------- work

# Operations of one ray query (8 node visits of 8 boxes, 4 triangles) and of one path vertex's shading.
_RAY_FLOPS, _VERTEX_FLOPS = 1000.0, 600.0


def _triangles(preset: int, scene_seed: int) -> int:
    b, _ = _builder(preset, scene_seed)
    a = b.arrays()
    mesh = [a.mesh_infos[i].index_offset for i in range(a.n_meshes)] + [a.n_indices]
    return sum((mesh[a.instances[i].mesh_id + 1] - mesh[a.instances[i].mesh_id]) // 3 for i in range(a.n_instances))


def _frame_work(pixels: int, photons: int, triangles: int) -> tuple[float, float]:
    """One frame: the scene's triangles read once (three corners), the sums of every pixel read and written,
    the image written; about four path vertices with a closest-hit and half a shadow ray each, one query per photon."""
    return 36.0 * triangles + 36.0 * pixels, pixels * 4.0 * (1.5 * _RAY_FLOPS + _VERTEX_FLOPS) + photons * _RAY_FLOPS


def work(case: dict) -> dict:
    kind = case["kind"]
    if kind == "grid":
        n = case["photons"]
        return {"bytes": 32.0 * n + 8.0 * n + 8.0 * (1 << case["hash_bits"]), "flops": 20.0 * n}
    if kind == "rays":
        return {"bytes": 48.0 * case["rays"] + 36.0 * _triangles(case["preset"], case["scene_seed"]),
                "flops": _RAY_FLOPS * case["rays"]}
    if kind == "batch":
        g = np.random.default_rng(case["scene_seed"])
        total = [0.0, 0.0]
        for k in range(case["scenes"]):
            w, h = (int(x) for x in g.integers(case["size_min"], case["size_max"] + 1, 2))
            f = _frame_work(w * h, case["photons"], _triangles(srt.PRESET_BATCH_RANDOM, case["scene_seed"] + k))
            total = [t + case["frames"] * x for t, x in zip(total, f)]
        return {"bytes": total[0], "flops": total[1]}
    preset = srt.PRESET_BATCH_RANDOM if kind == "animate" else case["preset"]
    by, fl = _frame_work(case["width"] * case["height"], case["photons"], _triangles(preset, case["scene_seed"]))
    n = case.get("frames", 1)
    return {"bytes": by * n, "flops": fl * n}


def exact(case: dict, seed: int):
    return None
