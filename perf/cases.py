"""The work that this framework is timed on, through its public entry points:
whole frames of the renderer, its passes one by one through the C ABI on the
data that a frame leaves them, ray sets, the denoiser, the display chain and
the radiance cache.

listed() gives the cases, draw(rng) another one of the same ranges,
prepare(case, seed) what a program holds before the call, run(state) one pass,
work(case) the bytes and operations that pass cannot do without, and
exact(case, seed) its outputs in 64 bits where they are a closed computation.
Scenes, sizes and settings are those of bench.py and of the tests. The hash
grid runs in its deterministic mode, so that the same inputs give the same
reservoirs.
"""
from __future__ import annotations

import ctypes as C
import functools
import math
import random

import numpy as np
import torch

import restir_b200 as rb
from restir_b200 import abi

SCENES = {"cornell": rb.SCENE_CORNELL, "courtyard": rb.SCENE_COURTYARD, "city": rb.SCENE_CITY}
RAY_KINDS = {"closest": rb.TRACE_CLOSEST, "any": rb.TRACE_ANY, "stackless": rb.TRACE_CLOSEST_STACKLESS,
             "watertight": rb.TRACE_CLOSEST_WATERTIGHT, "queue": rb.TRACE_CLOSEST_QUEUE}
HISTORY_FRAMES = 6  # frames rendered before a pass is taken out of one: its reservoirs and histories are settled
PATH_FRAMES = 32


def listed() -> list[dict]:
    return [
        # The smallest frame anyone renders: a Cornell box preview, bound by launches and latency.
        {"name": "frame_cornell_256", "kind": "frame", "scene": "cornell", "triangles": 36, "width": 256, "height": 256,
         "divisor": 1, "candidates": 1, "lights": 0, "rays": "hybrid", "cache": False},
        # The headline frame: 1080p, a million triangles, the default settings.
        {"name": "frame_city_1080p", "kind": "frame", "scene": "city", "triangles": 1_000_000, "width": 1920, "height": 1080,
         "divisor": 2, "candidates": 2, "lights": 64, "rays": "hybrid", "cache": False},
        # A mid-size interactive frame with the learned indirect light trained as it renders.
        {"name": "frame_courtyard_cache", "kind": "frame", "scene": "courtyard", "triangles": 100_000, "width": 1280,
         "height": 720, "divisor": 2, "candidates": 2, "lights": 64, "rays": "hybrid", "cache": True},
        # Indirect diffuse light of the headline frame: both resampling passes, called one by one by an engine.
        {"name": "gi_city_1080p", "kind": "gi", "scene": "city", "triangles": 1_000_000, "width": 1920, "height": 1080,
         "divisor": 2, "candidates": 2, "lights": 64, "rays": "hybrid"},
        # Many-light direct light of the headline frame, both passes.
        {"name": "di_city_1080p", "kind": "di", "scene": "city", "triangles": 1_000_000, "width": 1920, "height": 1080,
         "divisor": 2, "candidates": 2, "lights": 64, "rays": "hybrid"},
        # Visibility of the headline frame: the G-buffer's primary rays and the light's distance atlas.
        {"name": "primary_city_1080p", "kind": "primary", "scene": "city", "triangles": 1_000_000, "width": 1920,
         "height": 1080, "divisor": 2, "candidates": 2, "lights": 64, "rays": "hybrid"},
        # Glossy reflections in a window of odd size.
        {"name": "specular_courtyard_odd", "kind": "specular", "scene": "courtyard", "triangles": 100_000, "width": 1283,
         "height": 717, "divisor": 2, "candidates": 2, "lights": 64, "rays": "hybrid"},
        # A handful of rays, as picking or a probe update casts them: one launch's latency.
        {"name": "trace_cornell_1k", "kind": "trace", "scene": "cornell", "triangles": 36, "rays": 1000, "ray_kind": "closest"},
        # A baking or path tracing batch: a million incoherent nearest-hit rays through the ray queue.
        {"name": "trace_city_1m", "kind": "trace", "scene": "city", "triangles": 1_000_000, "rays": 1_000_000,
         "ray_kind": "queue"},
        # The denoiser at the resolution of a 1080p frame's indirect light.
        {"name": "denoise_960x540", "kind": "denoise", "width": 960, "height": 540, "levels": 5},
        # From the composite to the screen at 1440p: auto exposure, temporal anti-aliasing, tone mapping.
        {"name": "display_1440p", "kind": "display", "width": 2560, "height": 1440, "tonemapper": abi.TONEMAP_AGX},
        # A 1080p frame's use of the radiance cache: its queries and one training step.
        {"name": "cache_1080p", "kind": "cache", "queries": 2_073_600, "samples": 65_536},
    ]


def draw(rng: random.Random) -> dict:
    kind = rng.choice(["frame", "frame", "gi", "di", "primary", "specular", "trace", "trace", "denoise", "display", "cache"])
    if kind == "trace":
        scene, triangles = _draw_scene(rng)
        return {"kind": kind, "scene": scene, "triangles": triangles, "rays": _log_int(rng, 500, 1_000_000),
                "ray_kind": rng.choice(sorted(RAY_KINDS))}
    if kind == "denoise":
        width, height = _draw_size(rng, 120, 1920)
        return {"kind": kind, "width": width, "height": height, "levels": rng.randint(1, 5)}
    if kind == "display":
        width, height = _draw_size(rng, 120, 2560)
        return {"kind": kind, "width": width, "height": height, "tonemapper": rng.randint(0, 4)}
    if kind == "cache":
        return {"kind": kind, "queries": _log_int(rng, 1000, 2_000_000), "samples": _log_int(rng, 256, 65_536)}
    scene, triangles = _draw_scene(rng)
    width, height = _draw_size(rng, 160, 1920)
    # Full-resolution indirect light only for the smaller images.
    divisor = rng.choice([1, 2, 2, 4]) if width * height <= 500_000 else rng.choice([2, 2, 4])
    case = {"kind": kind, "scene": scene, "triangles": triangles, "width": width, "height": height, "divisor": divisor,
            "candidates": rng.choice([1, 2]), "lights": rng.choice([0, 16, 64]) if scene != "cornell" else rng.choice([0, 8]),
            "rays": rng.choice(["hybrid", "hybrid", "bvh"])}
    if kind == "frame":
        case["cache"] = rng.random() < 0.25 and width * height <= 1_000_000
    return case


def _log_int(rng: random.Random, low: int, high: int) -> int:
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def _draw_scene(rng: random.Random) -> tuple[str, int]:
    scene = rng.choice(["cornell", "courtyard", "city", "city"])
    return scene, 36 if scene == "cornell" else _log_int(rng, 20_000, 1_000_000 if scene == "city" else 200_000)


def _draw_size(rng: random.Random, low: int, high: int) -> tuple[int, int]:
    width = _log_int(rng, low, high)
    return width, max(64, int(width * rng.choice([0.5625, 0.5625, 0.75, 0.4375])))


# --- what a program holds -----------------------------------------------------------------------------


@functools.lru_cache(maxsize=3)
def _mesh(scene: str, triangles: int) -> rb.Mesh:
    return rb.Mesh.procedural(SCENES[scene], 0, triangles)


@functools.lru_cache(maxsize=3)
def _bvh(scene: str, triangles: int) -> rb.Bvh:
    return rb.Bvh(_mesh(scene, triangles), device=True)


def _generator(seed: int) -> torch.Generator:
    return torch.Generator(device="cuda").manual_seed(seed)


def _path(case: dict, mesh: rb.Mesh, seed: int) -> list:
    """Camera poses swaying about a pose near the scene's view."""
    rng = np.random.default_rng(seed)
    radius = mesh.desc.radius
    eye = np.array(mesh.desc.camera_eye, np.float64) + rng.uniform(-0.04, 0.04, 3) * radius * np.array([1.0, 0.25, 1.0])
    yaw = mesh.desc.camera_yaw + rng.uniform(-0.2, 0.2)
    pitch = mesh.desc.camera_pitch + rng.uniform(-0.04, 0.04)
    sway = rng.uniform(0.002, 0.006, 2)
    frames = []
    for k in range(PATH_FRAMES):
        a = 2.0 * math.pi * k / PATH_FRAMES
        at = eye + np.array([math.sin(a), 0.0, math.cos(a)]) * sway[0] * radius
        frames.append(rb.frame_input(mesh, case["width"], case["height"], eye=[float(x) for x in at],
                                     yaw=float(yaw + sway[1] * math.sin(a)), pitch=float(pitch)))
    return frames


def _renderer(case: dict, seed: int) -> tuple[rb.Renderer, list]:
    mesh = _mesh(case["scene"], case["triangles"])
    settings = rb.default_settings(mesh)
    settings.gi_divisor = case["divisor"]
    settings.initial_candidates = case["candidates"]
    settings.extra_lights = case["lights"]
    settings.ray_mode = rb.RAY_BVH if case["rays"] == "bvh" else rb.RAY_HYBRID
    settings.grid_mode = rb.GRID_DETERMINISTIC
    settings.radiance_cache = int(case.get("cache", False))
    renderer = rb.Renderer(settings)
    renderer.set_scene(mesh, use_scene_defaults=True)
    return renderer, _path(case, mesh, seed)


class _Frame:
    """A renderer after HISTORY_FRAMES frames, and the structs its last frame's passes read."""

    def __init__(self, case: dict, seed: int):
        self.renderer, self.path = _renderer(case, seed)
        for k in range(HISTORY_FRAMES):
            self.renderer.render(self.path[k])
        self.renderer.synchronize()
        self.params, self.plan, _ = self.renderer.last_frame()
        mesh = self.renderer.mesh
        self.gbuffer = abi.RestirGBuffer(*(self.at("gbuffer." + n) for n in ("albedo", "normal", "emissive", "shading_normal",
                                                                             "depth")))
        bvh_bytes = self.renderer.buffer("bvh")[1]
        self.scene = abi.RestirScene()
        self.scene.bvh = self.at("bvh")
        self.scene.node_count = (bvh_bytes // 16 - 4 * mesh.triangle_count) // 2
        self.scene.triangle_offset = 2 * self.scene.node_count
        self.scene.triangle_count = mesh.triangle_count
        self.scene.lights = self.at("lights")
        self.scene.light_count = self.params.di_light_count
        self.scene.triangle_normals = self.at("normals")
        self.scene.materials = self.at("materials")
        self.scene.material_count = mesh.desc.material_count
        # The targets alternate every frame, the first frame writing number 1.
        self.now = str(HISTORY_FRAMES % 2)
        self.before = str(1 - HISTORY_FRAMES % 2)
        self.atlas = self.at("shadow.atlas")
        self.surface = self.at("di.diffuse") if self.plan.di_active else self.at("black")
        self.history = abi.RestirGiHistory(self.at("gi.sample" + self.before), self.at("gi.receiver" + self.before),
                                           self.at("gi.normal" + self.before), self.at("filtered" + self.before),
                                           self.at("gi.moments" + self.before))
        self.pixels = self.params.width * self.params.height
        self.gi_pixels = self.params.gi_width * self.params.gi_height

    def at(self, name: str) -> int:
        return self.renderer.buffer(name)[0]


def _f32(rows: int, columns: int) -> torch.Tensor:
    return torch.zeros((rows, columns), dtype=torch.float32, device="cuda")


def _f16(rows: int) -> torch.Tensor:
    return torch.zeros((rows, 4), dtype=torch.float16, device="cuda")


def _u8(rows: int) -> torch.Tensor:
    return torch.zeros((rows, 4), dtype=torch.uint8, device="cuda")


def prepare(case: dict, seed: int) -> dict:
    return _PREPARE[case["kind"]](case, seed)


def run(state: dict):
    return _RUN[state["kind"]](state)


# --- whole frames -------------------------------------------------------------------------------------


class _Target:
    """One of a renderer's buffers; tensors made of it keep the renderer alive."""

    def __init__(self, renderer: rb.Renderer, name: str):
        pointer, size = renderer.buffer(name)
        self.renderer = renderer
        self.__cuda_array_interface__ = {"shape": (size,), "typestr": "|u1", "data": (pointer, False), "version": 3}


def _prepare_frame(case: dict, seed: int) -> dict:
    renderer, path = _renderer(case, seed)
    for k in range(HISTORY_FRAMES):
        renderer.render(path[k])
    renderer.synchronize()

    def view(name, dtype, count):
        return torch.as_tensor(_Target(renderer, name), device="cuda").view(dtype)[:count]

    pixels = case["width"] * case["height"]
    outputs = {"hdr": view("hdr", torch.float16, 4 * pixels), "display": view("display", torch.uint8, 4 * pixels),
               "depth": view("gbuffer.depth", torch.float32, pixels)}
    if renderer.last_frame()[1].di_active:
        outputs["diffuse"] = view("di.diffuse", torch.float16, 4 * pixels)
        outputs["specular"] = view("di.specular", torch.float16, 4 * pixels)
    return {"kind": "frame", "renderer": renderer, "path": path, "next": HISTORY_FRAMES, "outputs": outputs}


def _run_frame(state: dict):
    state["renderer"].render(state["path"][state["next"] % PATH_FRAMES])
    state["next"] += 1
    return state["outputs"]


# --- single passes ------------------------------------------------------------------------------------


def _prepare_gi(case: dict, seed: int) -> dict:
    f = _Frame(case, seed)
    n = f.gi_pixels
    out = {"sample": _f32(n, 4), "receiver": _f32(n, 4), "normal": _f32(n, 4), "color": _f16(n), "moments": _f16(n)}
    size = rb.load().restir_gi_temporal_workspace_bytes(f.params)
    return {"kind": "gi", "frame": f, "out": out, "workspace": torch.zeros(size, dtype=torch.uint8, device="cuda"),
            "reservoirs": abi.RestirGiReservoirs(*(out[k].data_ptr() for k in ("sample", "receiver", "normal"))),
            "grid": f.at("grid" + f.before), "grid_now": f.at("grid" + f.now)}


def _run_gi(state: dict):
    f, out, lib = state["frame"], state["out"], rb.load()
    rb.check(lib.restir_gi_temporal_wavefront(f.params, f.scene, f.gbuffer, f.history, state["grid"], f.atlas, f.surface,
                                              state["reservoirs"], state["workspace"].data_ptr(), state["workspace"].numel(),
                                              None), "restir_gi_temporal_wavefront")
    rb.check(lib.restir_gi_spatial(f.params, f.scene, f.gbuffer, state["reservoirs"], state["grid_now"], f.history, f.atlas,
                                   f.surface, out["color"].data_ptr(), out["moments"].data_ptr(), None), "restir_gi_spatial")
    return out


def _prepare_di(case: dict, seed: int) -> dict:
    f = _Frame(case, seed)
    n = f.pixels
    out = {"sample": _f32(n, 4), "receiver": _f32(n, 4), "normal": _f16(n), "diffuse": _f16(n), "specular": _f16(n)}
    previous = abi.RestirDiReservoirs(*(f.at("di." + k + f.before) for k in ("sample", "receiver", "normal")))
    return {"kind": "di", "frame": f, "out": out, "previous": previous,
            "reservoirs": abi.RestirDiReservoirs(*(out[k].data_ptr() for k in ("sample", "receiver", "normal")))}


def _run_di(state: dict):
    f, out, lib = state["frame"], state["out"], rb.load()
    rb.check(lib.restir_di_temporal(f.params, f.scene, f.gbuffer, state["previous"], state["reservoirs"], None),
             "restir_di_temporal")
    rb.check(lib.restir_di_spatial(f.params, f.scene, f.gbuffer, state["reservoirs"], out["diffuse"].data_ptr(),
                                   out["specular"].data_ptr(), None), "restir_di_spatial")
    return out


def _prepare_primary(case: dict, seed: int) -> dict:
    f = _Frame(case, seed)
    n, face = f.pixels, f.params.shadow_face_size
    out = {"albedo": _u8(n), "normal": _u8(n), "emissive": _f16(n), "shading_normal": _u8(n), "depth": _f32(n, 1),
           "atlas": _f32(6 * face, face)}
    targets = abi.RestirGBuffer(*(out[k].data_ptr() for k in ("albedo", "normal", "emissive", "shading_normal", "depth")))
    return {"kind": "primary", "frame": f, "out": out, "targets": targets}


def _run_primary(state: dict):
    f, out, lib = state["frame"], state["out"], rb.load()
    rb.check(lib.restir_shadow_atlas(f.params, f.scene, out["atlas"].data_ptr(), None), "restir_shadow_atlas")
    rb.check(lib.restir_gbuffer_primary(f.params, f.scene, state["targets"], None), "restir_gbuffer_primary")
    return out


def _prepare_specular(case: dict, seed: int) -> dict:
    f = _Frame(case, seed)
    size = rb.load().restir_gi_specular_workspace_bytes(f.params)
    return {"kind": "specular", "frame": f, "out": _f16(f.gi_pixels), "hdr": f.at("hdr"),
            "previous": f.at("specular" + f.before), "workspace": torch.zeros(size, dtype=torch.uint8, device="cuda")}


def _run_specular(state: dict):
    f, out = state["frame"], state["out"]
    rb.check(rb.load().restir_gi_specular_wavefront(f.params, f.scene, f.gbuffer, f.history, f.atlas, f.surface, state["hdr"],
                                                    state["previous"], out.data_ptr(), state["workspace"].data_ptr(),
                                                    state["workspace"].numel(), None), "restir_gi_specular_wavefront")
    return out


# --- ray sets -----------------------------------------------------------------------------------------


def _rays(case: dict, seed: int) -> torch.Tensor:
    """Origins over the scene's box, directions over the sphere: (n, 8) float32."""
    d, n, g = _mesh(case["scene"], case["triangles"]).desc, case["rays"], _generator(seed)
    low = torch.tensor(list(d.bounds_min), device="cuda")
    high = torch.tensor(list(d.bounds_max), device="cuda")
    rays = torch.zeros((n, 8), dtype=torch.float32, device="cuda")
    rays[:, 0:3] = low + (high - low) * torch.rand((n, 3), generator=g, device="cuda")
    rays[:, 3] = 4.0 * d.radius
    rays[:, 4:7] = torch.nn.functional.normalize(torch.randn((n, 3), generator=g, device="cuda"), dim=1)
    return rays


def _prepare_trace(case: dict, seed: int) -> dict:
    bvh = _bvh(case["scene"], case["triangles"])
    rows = torch.from_numpy(bvh.data).cuda()
    scene = abi.RestirScene()
    scene.bvh = rows.data_ptr()
    scene.node_count = bvh.desc.node_count
    scene.triangle_offset = bvh.desc.triangle_offset
    scene.triangle_count = bvh.desc.triangle_count
    n = case["rays"]
    return {"kind": "trace", "rows": rows, "scene": scene, "rays": _rays(case, seed), "ray_kind": RAY_KINDS[case["ray_kind"]],
            "triangle": torch.zeros(n, dtype=torch.int32, device="cuda"), "distance": torch.zeros(n, device="cuda")}


def _run_trace(state: dict):
    rb.check(rb.load().restir_trace(None, state["scene"], state["rays"].data_ptr(), state["triangle"].data_ptr(),
                                    state["distance"].data_ptr(), state["rays"].shape[0], state["ray_kind"], None),
             "restir_trace")
    return {"triangle": state["triangle"], "distance": state["distance"]}


def _exact_trace(case: dict, seed: int):
    if case["scene"] != "cornell" or case["ray_kind"] == "any":
        return None  # too many triangles to try them all; any hit may be reported
    vertices = torch.from_numpy(_mesh("cornell", case["triangles"]).positions()).cuda().double().reshape(-1, 3, 3)
    distances = []
    for rays in _rays(case, seed).double().split(100_000):
        o, d, best = rays[:, None, 0:3], rays[:, None, 4:7], rays[:, 3].clone()
        v0, e1, e2 = vertices[None, :, 0], (vertices[:, 1] - vertices[:, 0])[None], (vertices[:, 2] - vertices[:, 0])[None]
        p = torch.linalg.cross(d.expand(-1, e2.shape[1], -1), e2.expand(d.shape[0], -1, -1))
        inverse = 1.0 / (e1 * p).sum(-1)
        s = o - v0
        u = (s * p).sum(-1) * inverse
        q = torch.linalg.cross(s, e1.expand_as(s))
        v = (d * q).sum(-1) * inverse
        t = (e2 * q).sum(-1) * inverse
        hit = (u >= 0) & (v >= 0) & (u + v <= 1) & (t > 0)
        distances.append(torch.minimum(best, torch.where(hit, t, torch.inf).amin(1)))
    return {"triangle": None, "distance": torch.cat(distances)}


# --- denoiser -----------------------------------------------------------------------------------------

DENOISE_SCALE = 1.0


def _denoise_inputs(case: dict, seed: int) -> dict:
    """A room of flat walls at several depths and angles, some background, noisy
    light with the moments of 1 to 16 frames."""
    w, h, g = case["width"], case["height"], _generator(seed)
    y, x = torch.meshgrid(torch.arange(h, device="cuda"), torch.arange(w, device="cuda"), indexing="ij")
    wall = (x * 5 // w + 3 * (y * 4 // h) + seed) % 5
    normals = torch.tensor([[0, 0, -1], [0, 1, 0], [1, 0, 0], [-0.6, 0, -0.8], [0, 0.8, -0.6]], device="cuda",
                           dtype=torch.float32)
    n = normals[wall]
    receiver = torch.zeros((h, w, 4), device="cuda")
    receiver[..., 0] = (x / w - 0.5) * 3.0
    receiver[..., 1] = (0.5 - y / h) * 2.0
    # Depth along each wall's plane, with the noise of decoded positions.
    receiver[..., 2] = wall * 0.4 - receiver[..., 0] * n[..., 0] - receiver[..., 1] * 0.3 * n[..., 1]
    receiver[..., :3] += 1e-3 * torch.randn((h, w, 3), generator=g, device="cuda")
    normal = torch.zeros((h, w, 4), device="cuda")
    normal[..., :3] = n
    background = torch.rand((h // 16 + 1, w // 16 + 1), generator=g, device="cuda") < 0.06
    background = background.repeat_interleave(16, 0).repeat_interleave(16, 1)[:h, :w]
    normal[background] = 0.0
    color = torch.exp(0.8 * torch.randn((h, w, 4), generator=g, device="cuda") - 1.0)
    length = torch.floor(1.0 + 15.0 * torch.rand((h, w), generator=g, device="cuda") ** 0.5)
    color[..., 3] = length
    lum = color[..., 0] * 0.2126 + color[..., 1] * 0.7152 + color[..., 2] * 0.0722
    moments = torch.stack([lum, lum * lum * (1.0 + torch.rand((h, w), generator=g, device="cuda")), length,
                           torch.zeros_like(lum)], -1)
    return {"color": color.half(), "moments": moments.half(), "receiver": receiver, "normal": normal}


def _prepare_denoise(case: dict, seed: int) -> dict:
    inputs = _denoise_inputs(case, seed)
    params = abi.RestirParams()
    params.gi_width, params.gi_height, params.scene_scale = case["width"], case["height"], DENOISE_SCALE
    n = case["width"] * case["height"]
    return {"kind": "denoise", "inputs": inputs, "params": params, "levels": case["levels"],
            "filters": [_f16(n) for _ in range(case["levels"] + 1)]}


def _run_denoise(state: dict):
    lib, p, filters = rb.load(), state["params"], state["filters"]
    color, moments, receiver, normal = (state["inputs"][k].data_ptr() for k in ("color", "moments", "receiver", "normal"))
    rb.check(lib.restir_svgf_variance(p, color, moments, receiver, normal, filters[0].data_ptr(), None), "restir_svgf_variance")
    for level in range(state["levels"]):
        rb.check(lib.restir_svgf_atrous(p, 1 << level, filters[level].data_ptr(), receiver, normal,
                                        filters[level + 1].data_ptr(), None), "restir_svgf_atrous")
    # The frame's history is the first level's output.
    return {"history": filters[1], "filtered": filters[-1]}


def _shift(image: torch.Tensor, dx: int, dy: int) -> tuple[torch.Tensor, torch.Tensor]:
    """image at (x + dx, y + dy), clamped to the edge, and whether that is inside."""
    h, w = image.shape[:2]
    y = torch.arange(h, device=image.device) + dy
    x = torch.arange(w, device=image.device) + dx
    inside = ((y >= 0) & (y < h))[:, None] & ((x >= 0) & (x < w))[None, :]
    return image[y.clamp(0, h - 1)][:, x.clamp(0, w - 1)], inside


def _luminance(c: torch.Tensor) -> torch.Tensor:
    return (c[..., :3] * torch.tensor([0.2126, 0.7152, 0.0722], dtype=c.dtype, device=c.device)).sum(-1)


def _exact_denoise(case: dict, seed: int):
    inputs = {k: v.double() for k, v in _denoise_inputs(case, seed).items()}
    position, raw = inputs["receiver"][..., :3], inputs["normal"][..., :3]
    valid = (raw * raw).sum(-1) >= 0.5
    unit = torch.nn.functional.normalize(raw, dim=-1)

    def geometry(dx, dy):
        other, inside = _shift(torch.cat([position, unit, valid[..., None].double()], -1), dx, dy)
        plane = ((other[..., :3] - position) * unit).sum(-1).abs() / (0.02 * DENOISE_SCALE)
        weight = torch.exp(-plane) * (unit * other[..., 3:6]).sum(-1).clamp(min=0.0) ** 64
        return torch.where(inside & (other[..., 6] > 0.5), weight, 0.0)

    moments, length = inputs["moments"], inputs["moments"][..., 2]
    sums = torch.zeros_like(moments[..., :2])
    total = torch.zeros_like(length)
    for dy in range(-3, 4):
        for dx in range(-3, 4):
            weight = geometry(dx, dy)
            sums += _shift(moments, dx, dy)[0][..., :2] * weight[..., None]
            total += weight
    mean = sums / total.clamp(min=0.0001)[..., None]
    short = (mean[..., 1] - mean[..., 0] ** 2).clamp(min=0.0) * (4.0 / length.clamp(min=1.0))
    long = (moments[..., 1] - moments[..., 0] ** 2).clamp(min=0.0)
    image = torch.cat([inputs["color"][..., :3], torch.where(length >= 4.0, long, short)[..., None]], -1)
    image = torch.where(valid[..., None], image, 0.0)
    outputs = []
    spline = {0: 0.375, 1: 0.25, 2: 0.0625}
    for level in range(case["levels"]):
        step = 1 << level
        variance = torch.zeros_like(length)
        for dy in (-1, 0, 1):
            for dx in (-1, 0, 1):
                variance += _shift(image, dx, dy)[0][..., 3] * (0.5 if dx == 0 else 0.25) * (0.5 if dy == 0 else 0.25)
        scale = 1.0 / (4.0 * variance.clamp(min=0.0).sqrt() + 0.0001)
        center = _luminance(image)
        color, spread = torch.zeros_like(image[..., :3]), torch.zeros_like(length)
        total = torch.zeros_like(length)
        for dy in range(-2, 3):
            for dx in range(-2, 3):
                tap, inside = _shift(image, dx * step, dy * step)
                weight = inside * (spline[abs(dx)] * spline[abs(dy)])
                if dx or dy:
                    weight = weight * geometry(dx * step, dy * step) * torch.exp(-(_luminance(tap) - center).abs() * scale)
                color += tap[..., :3] * weight[..., None]
                spread += tap[..., 3] * weight * weight
                total += weight
        image = torch.cat([color / total[..., None], (spread / (total * total))[..., None]], -1)
        image = torch.where(valid[..., None], image, 0.0)
        outputs.append(image.reshape(-1, 4))
    return {"history": outputs[0], "filtered": outputs[-1]}


# --- display ------------------------------------------------------------------------------------------


def _perspective(eye, aspect: float) -> np.ndarray:
    """A row-major view-projection looking at the origin (clip = M v, NDC depth in [0, 1])."""
    eye = np.asarray(eye, np.float64)
    forward = -eye / np.linalg.norm(eye)
    right = np.cross(forward, [0.0, 1.0, 0.0])
    right /= np.linalg.norm(right)
    view = np.eye(4)
    view[0, :3], view[1, :3], view[2, :3] = right, np.cross(right, forward), forward
    view[:3, 3] = -view[:3, :3] @ eye
    f, near, far = 1.0 / math.tan(0.5), 0.05, 50.0
    projection = np.zeros((4, 4))
    projection[0, 0], projection[1, 1], projection[3, 2] = f / aspect, f, 1.0
    projection[2, 2], projection[2, 3] = far / (far - near), -near * far / (far - near)
    return projection @ view


def _display_inputs(case: dict, seed: int) -> dict:
    """A composite and last frame's output of a view that moved a little, with some background."""
    w, h, g = case["width"], case["height"], _generator(seed)
    base = torch.exp(1.5 * torch.randn((h // 4 + 2, w // 4 + 2, 3), generator=g, device="cuda") - 1.0)
    base = base.repeat_interleave(4, 0).repeat_interleave(4, 1)[:h, :w]
    background = (torch.rand((h // 8 + 1, w // 8 + 1), generator=g, device="cuda") < 0.1).repeat_interleave(8, 0)
    background = background.repeat_interleave(8, 1)[:h, :w]
    images = []
    for _ in range(2):
        image = torch.ones((h, w, 4), device="cuda")
        image[..., :3] = base * torch.exp(0.3 * torch.randn((h, w, 3), generator=g, device="cuda"))
        image[..., 3] = (~background).float()
        images.append(image.half())
    depth = 0.95 + 0.045 * torch.rand((h, w), generator=g, device="cuda")
    depth[background] = 1.0
    move = np.random.default_rng(seed).uniform(-0.03, 0.03, 3)
    now = _perspective(np.array([0.3, 0.5, -3.0]), w / h).astype(np.float32)
    return {"hdr": images[0], "history": images[1], "depth": depth, "inverse": np.linalg.inv(now.astype(np.float64)).astype(np.float32),
            "previous": _perspective(np.array([0.3, 0.5, -3.0]) + move, w / h).astype(np.float32)}


def _prepare_display(case: dict, seed: int) -> dict:
    inputs = _display_inputs(case, seed)
    params = abi.RestirDisplayParams()
    params.inv_view_proj[:] = [float(v) for v in inputs["inverse"].reshape(-1)]
    params.previous_view_proj[:] = [float(v) for v in inputs["previous"].reshape(-1)]
    params.width, params.height = case["width"], case["height"]
    params.taa_history_valid, params.taa, params.auto_exposure = 1.0, 1.0, 1.0
    params.exposure_adapt, params.tonemapper = 0.05, float(case["tonemapper"])
    n = case["width"] * case["height"]
    return {"kind": "display", "inputs": inputs, "params": params, "taa": _f16(n), "display": _u8(n),
            "exposure": torch.zeros(1, dtype=torch.int32, device="cuda")}


def _run_display(state: dict):
    i = state["inputs"]
    rb.check(rb.load().restir_display(state["params"], i["hdr"].data_ptr(), i["depth"].data_ptr(), i["history"].data_ptr(),
                                      state["taa"].data_ptr(), state["exposure"].data_ptr(), None, None,
                                      state["display"].data_ptr(), None), "restir_display")
    return {"taa": state["taa"], "display": state["display"], "exposure": state["exposure"]}


def _exact_display(case: dict, seed: int):
    """The temporal anti-aliasing target; the display's bytes and the exposure's bits have no such value."""
    i = _display_inputs(case, seed)
    w, h = case["width"], case["height"]
    hdr, history, depth = i["hdr"].double(), i["history"].double(), i["depth"].double()
    to_ycocg = torch.tensor([[0.25, 0.5, 0.25], [0.5, 0.0, -0.5], [-0.25, 0.5, -0.25]], dtype=torch.float64, device="cuda")

    def ycocg(c):
        return (c / (1.0 + _luminance(c))[..., None]) @ to_ycocg.T

    y, x = torch.meshgrid(torch.arange(h, device="cuda"), torch.arange(w, device="cuda"), indexing="ij")
    texel = torch.tensor([1.0 / w, 1.0 / h], dtype=torch.float64, device="cuda")
    uv = torch.stack([x + 0.5, y + 0.5], -1).double() * texel
    compressed = ycocg(hdr[..., :3])
    total, squares = torch.zeros_like(compressed), torch.zeros_like(compressed)
    nearest, nearest_uv = torch.ones_like(depth), uv.clone()
    for dy in (-1, 0, 1):
        for dx in (-1, 0, 1):
            c = _shift(compressed, dx, dy)[0]
            d = _shift(depth, dx, dy)[0]
            total, squares = total + c, squares + c * c
            closer = d < nearest
            nearest = torch.where(closer, d, nearest)
            nearest_uv = torch.where(closer[..., None], uv + torch.tensor([dx, dy], device="cuda") * texel, nearest_uv)
    inverse = torch.from_numpy(i["inverse"]).cuda().double()
    previous = torch.from_numpy(i["previous"]).cuda().double()
    clip = torch.stack([nearest_uv[..., 0] * 2 - 1, 1 - nearest_uv[..., 1] * 2, nearest, torch.ones_like(nearest)], -1)
    world = clip @ inverse.T
    past_clip = (world / world[..., 3:]) @ previous.T
    past_uv = torch.stack([past_clip[..., 0], -past_clip[..., 1]], -1) / past_clip[..., 3:] * 0.5 + 0.5 + (uv - nearest_uv)
    keep = (past_clip[..., 3] <= 1e-4) | (past_uv < 0).any(-1) | (past_uv > 1).any(-1)

    def bilinear(u, v):
        px, py = u * w - 0.5, v * h - 0.5
        bx, by = px.floor(), py.floor()
        fx, fy = (px - bx)[..., None], (py - by)[..., None]
        x0, x1 = bx.clamp(0, w - 1).long(), (bx + 1).clamp(0, w - 1).long()
        y0, y1 = by.clamp(0, h - 1).long(), (by + 1).clamp(0, h - 1).long()
        top = history[y0, x0, :3] * (1 - fx) + history[y0, x1, :3] * fx
        bottom = history[y1, x0, :3] * (1 - fx) + history[y1, x1, :3] * fx
        return top * (1 - fy) + bottom * fy

    position = past_uv / texel
    center = (position - 0.5).floor() + 0.5
    f = position - center
    w0 = f * (-0.5 + f * (1.0 - 0.5 * f))
    w1 = 1.0 + f * f * (-2.5 + 1.5 * f)
    w2 = f * (0.5 + f * (2.0 - 1.5 * f))
    w3 = f * f * (-0.5 + 0.5 * f)
    w12 = w1 + w2
    uv0, uv3, uv12 = (center - 1.0) * texel, (center + 2.0) * texel, (center + w2 / w12) * texel
    taps = [(uv12[..., 0], uv0[..., 1], w12[..., 0] * w0[..., 1]), (uv0[..., 0], uv12[..., 1], w0[..., 0] * w12[..., 1]),
            (uv12[..., 0], uv12[..., 1], w12[..., 0] * w12[..., 1]), (uv3[..., 0], uv12[..., 1], w3[..., 0] * w12[..., 1]),
            (uv12[..., 0], uv3[..., 1], w12[..., 0] * w3[..., 1])]
    color = sum(bilinear(u, v) * weight[..., None] for u, v, weight in taps)
    past = ycocg((color / sum(weight for _, _, weight in taps)[..., None]).clamp(min=0.0))
    mean = total / 9.0
    extent = (squares / 9.0 - mean * mean).clamp(min=0.0).sqrt() * 1.25
    offset = past - mean
    largest = (offset / extent.clamp(min=0.00001)).abs().amax(-1, keepdim=True)
    past = torch.where(largest > 1.0, mean + offset / largest, past)
    rgb = torch.stack([past[..., 0] + past[..., 1] - past[..., 2], past[..., 0] + past[..., 2],
                       past[..., 0] - past[..., 1] - past[..., 2]], -1)
    blended = rgb * 0.9 + hdr[..., :3] / (1.0 + _luminance(hdr))[..., None] * 0.1
    result = blended / (1.0 - _luminance(blended)).clamp(min=0.0001)[..., None]
    result = torch.where(keep[..., None], hdr[..., :3], result)
    return {"taa": torch.cat([result, hdr[..., 3:]], -1).reshape(-1, 4), "display": None, "exposure": None}


# --- radiance cache -----------------------------------------------------------------------------------


def _cache_inputs(case: dict, seed: int) -> dict:
    """A cache as training leaves one, the frame's queries and a training batch."""
    g = _generator(seed)

    def queries(n):
        q = torch.zeros((n, 16), device="cuda")
        q[:, 0:3] = 2.0 * torch.rand((n, 3), generator=g, device="cuda") - 1.0
        q[:, 3] = torch.rand(n, generator=g, device="cuda")
        for column in (4, 8):
            q[:, column:column + 3] = torch.nn.functional.normalize(torch.randn((n, 3), generator=g, device="cuda"), dim=1)
        q[:, 7] = 1.0
        q[:, 12:15] = 0.05 + 0.9 * torch.rand((n, 3), generator=g, device="cuda")
        return q

    weights = 0.18 * torch.randn(abi.CACHE_WEIGHTS, generator=g, device="cuda")
    weights[4 * 4096 + 3 * 64:] = 0.0  # the output rows that are not used
    table = 0.2 * torch.randn((abi.CACHE_LEVELS << 18, abi.CACHE_FEATURES), generator=g, device="cuda")
    targets = torch.ones((case["samples"], 4), device="cuda")
    targets[:, :3] = torch.exp(torch.randn((case["samples"], 3), generator=g, device="cuda") - 1.0)
    return {"weights": weights, "table": table, "queries": queries(case["queries"]), "batch": queries(case["samples"]),
            "targets": targets}


def _cache_config() -> abi.RestirCacheConfig:
    return rb.cache_config(bounds_min=(-1.0, -1.0, -1.0), bounds_max=(1.0, 1.0, 1.0))


def _prepare_cache(case: dict, seed: int) -> dict:
    inputs = _cache_inputs(case, seed)
    cache = rb.RadianceCache(_cache_config())
    cache.region("weights", torch.float32, abi.CACHE_WEIGHTS).copy_(inputs["weights"])
    cache.region("weights_bf16", torch.bfloat16, abi.CACHE_WEIGHTS).copy_(inputs["weights"])
    cache.region("table", torch.float32, inputs["table"].numel()).copy_(inputs["table"].reshape(-1))
    cache.region("table_half", torch.float16, inputs["table"].numel()).copy_(inputs["table"].reshape(-1))
    values = _f16(case["queries"])
    return {"kind": "cache", "cache": cache, "queries": inputs["queries"], "batch": inputs["batch"],
            "targets": inputs["targets"], "values": values,
            "out": {"values": values, "weights": cache.region("weights", torch.float32, abi.CACHE_WEIGHTS),
                    "weight_gradient": cache.region("weight_grad", torch.float32, abi.CACHE_WEIGHTS),
                    "table_gradient": cache.region("table_grad", torch.float32, inputs["table"].numel())}}


def _run_cache(state: dict):
    state["cache"].query(state["queries"], state["values"])
    state["cache"].train(state["batch"], state["targets"])
    return state["out"]


def _cache_network(table: torch.Tensor, weights: torch.Tensor, queries: torch.Tensor) -> torch.Tensor:
    """The cache's outputs: the hash encoding and the network in 64 bits."""
    layout = rb.cache_layout(_cache_config())
    unit = ((queries[:, 0:3].double() + 1.0) / 2.0).clamp(0.0, 1.0)
    features = []
    for level in range(abi.CACHE_LEVELS):
        scale = int(layout.level_scale[level])
        at = unit * scale
        cell = at.floor().long().clamp(max=scale - 1)
        part = at - cell
        bricks = (scale + 2) // 2
        value = 0.0
        for corner in range(8):
            step = torch.tensor([corner & 1, (corner >> 1) & 1, corner >> 2], device="cuda")
            p = cell + step
            weight = torch.where(step.bool(), part, 1.0 - part).prod(-1, keepdim=True)
            b = p // 2
            if layout.level_dense[level]:
                brick = b[:, 0] + b[:, 1] * bricks + b[:, 2] * bricks * bricks
            else:
                brick = (b[:, 0] ^ ((b[:, 1] * 2654435761) & 0xffffffff) ^ ((b[:, 2] * 805459861) & 0xffffffff)) \
                    % (layout.entries // 8)
            index = brick * 8 + (p[:, 0] % 2) + 2 * (p[:, 1] % 2) + 4 * (p[:, 2] % 2)
            value = value + weight * table[level * layout.entries + index]
        features.append(value)
    q = queries.double()
    x = torch.cat(features + [q[:, 8:11], q[:, 4:7], q[:, 3:4], q[:, 12:15], torch.ones_like(q[:, :1]),
                              torch.zeros((q.shape[0], 21), dtype=torch.float64, device="cuda")], -1)
    for layer in range(4):
        x = (x @ weights[layer * 4096:(layer + 1) * 4096].reshape(64, 64).T).clamp(min=0.0)
    return x @ weights[4 * 4096:].reshape(16, 64).T


def _exact_cache(case: dict, seed: int):
    inputs = _cache_inputs(case, seed)
    # The network computes with the 16-bit copies of its parameters.
    table = inputs["table"].half().double()
    weights = inputs["weights"].bfloat16().double()
    values = []
    with torch.no_grad():
        for part in inputs["queries"].split(100_000):
            y = _cache_network(table, weights, part)[:, :3].clamp(min=0.0)
            values.append(torch.cat([y, torch.ones_like(y[:, :1])], -1))
    table.requires_grad_()
    weights.requires_grad_()
    targets = inputs["targets"].double()
    for part, target in zip(inputs["batch"].split(16_384), targets.split(16_384)):
        y = _cache_network(table, weights, part)[:, :3]
        loss = ((y - target[:, :3]) ** 2 / (y.detach() ** 2 + 0.01) * target[:, 3:]).sum() / (3 * case["samples"])
        loss.backward()
    return {"values": torch.cat(values), "weights": None, "weight_gradient": weights.grad,
            "table_gradient": table.grad.reshape(-1)}


# --- what a pass cannot do without --------------------------------------------------------------------


def _scene_bytes(case: dict) -> float:
    """The acceleration structure's rows, each read once: about 0.96 nodes of 32 bytes and 64 bytes a triangle."""
    return case["triangles"] * (0.96 * 2 * 32 + 64) / 2.0


def work(case: dict) -> dict:
    kind = case["kind"]
    if kind == "trace":
        # A ray and its hit; a walk's box and triangle tests, about 40 nodes of 23 operations at least.
        depth = math.log2(max(case["triangles"], 2)) * 2.0
        return {"bytes": case["rays"] * 40.0 + min(_scene_bytes(case), case["rays"] * depth * 32.0),
                "flops": case["rays"] * depth * 23.0}
    if kind == "cache":
        network = 2.0 * (4 * 64 * 64 + 3 * 64)
        table = (abi.CACHE_LEVELS << 18) * abi.CACHE_FEATURES
        # Rows and gathers of the queries and samples; Adam reads and writes every parameter and moment.
        return {"bytes": case["queries"] * (64.0 + 512.0 + 8.0) + case["samples"] * (64.0 + 2 * 512.0 + 16.0) + table * 30.0,
                "flops": case["queries"] * network + 3.0 * case["samples"] * network}
    pixels = case["width"] * case["height"]
    if kind == "denoise":
        return {"bytes": pixels * (16 + 32 + 8 + case["levels"] * (8 + 32 + 8.0)), "flops": pixels * (60 + case["levels"] * 24 * 40.0)}
    if kind == "display":
        return {"bytes": pixels * 32.0, "flops": pixels * 400.0}
    gi = pixels / case["divisor"] ** 2
    scene = _scene_bytes(case)
    # Image reads and writes of each pass per pixel, and a walk of each ray it cannot do without.
    depth = math.log2(case["triangles"] + 2) * 2.0 * 23.0
    atlas = 6 * 512 * 512
    passes = {
        "primary": (pixels * 24.0 + atlas * 4.0 + scene, (pixels + atlas) * depth),
        "di": (pixels * (96 + 72.0) + scene, pixels * (2 * depth + 2000.0)),
        "gi": (gi * (116 + 124.0) + scene, gi * ((case["candidates"] + 2) * depth + 2000.0)),
        "specular": (gi * 96.0 + scene, gi * (depth + 500.0)),
    }
    if kind != "frame":
        return {"bytes": passes[kind][0], "flops": passes[kind][1]}
    total_bytes = sum(b for b, _ in passes.values()) - 3 * scene + gi * (20 + 56 + 5 * 48.0) + pixels * (50 + 32.0)
    total_flops = sum(f for _, f in passes.values()) + gi * 5000.0 + pixels * 800.0
    if case["cache"]:
        cached = work({"kind": "cache", "queries": int(gi * (case["candidates"] + 2)), "samples": 65_536})
        total_bytes, total_flops = total_bytes + cached["bytes"], total_flops + cached["flops"]
    return {"bytes": total_bytes, "flops": total_flops}


def exact(case: dict, seed: int):
    """None for the rendering passes: their outputs follow from discrete choices (hits, resampled
    neighbours) that 64 bits would make otherwise."""
    fn = {"trace": _exact_trace, "denoise": _exact_denoise, "display": _exact_display, "cache": _exact_cache}.get(case["kind"])
    return fn(case, seed) if fn is not None else None


_PREPARE = {"frame": _prepare_frame, "gi": _prepare_gi, "di": _prepare_di, "primary": _prepare_primary,
            "specular": _prepare_specular, "trace": _prepare_trace, "denoise": _prepare_denoise, "display": _prepare_display,
            "cache": _prepare_cache}
_RUN = {"frame": _run_frame, "gi": _run_gi, "di": _run_di, "primary": _run_primary, "specular": _run_specular,
        "trace": _run_trace, "denoise": _run_denoise, "display": _run_display, "cache": _run_cache}
