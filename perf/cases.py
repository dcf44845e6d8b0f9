"""Timed cases of the atmosphere renderer: what a frame loop, a LUT baker and a
surrogate trainer call, over their range of sizes.

A case is a dict of plain values with a ``kind``:

* ``frame``     the drop-in frame of the reference's scheduler: per camera
                ``update`` (a moving camera rebuilds the sky-view LUT),
                ``prepare_frame``, ``composite``;
* ``fused``     ``update`` and ``render_frame`` (lighting, land and ocean
                shading and the composite in one pass);
* ``surrogate`` ``update`` and ``composite_surrogate`` (the learned composite);
* ``sky``       ``sky_pixels``: a sky radiance image, marched, by the sky
                network or from the LUT;
* ``luts``      one set of the four LUTs, baked and read back as fields;
* ``batch``     many sky-view and aerial LUTs in one ``BatchedLutBuilder.build``;
* ``train``     one optimiser step of a surrogate network;
* ``evaluate``  a held-out set through a network in FP32 and in BF16;
* ``gbuffer``   terrain raster and ocean coverage: the frame's G-buffer;
* ``post``      the display post-process;
* ``display``   a whole frame, from terrain patches to the display image.

``exact`` restates the reference's algorithm in 64-bit torch.
"""

from __future__ import annotations

import dataclasses
import math
import sys
from pathlib import Path

import numpy as np
import torch

sys.path.insert(0, str(Path(__file__).resolve().parents[1] / "planet-real-time-render_gb300"))

from planet_renderer_gb300 import camera  # noqa: E402
from planet_renderer_gb300.atmosphere import AtmosphereRenderer  # noqa: E402
from planet_renderer_gb300.atmosphere import config as atm_config  # noqa: E402
from planet_renderer_gb300.atmosphere.batch import BatchedLutBuilder  # noqa: E402
from planet_renderer_gb300.atmosphere.mlp import HIDDEN, Mlp, layer_shapes  # noqa: E402
from planet_renderer_gb300.atmosphere.surrogate import Surrogate  # noqa: E402
from planet_renderer_gb300.atmosphere.workloads import (EARTH_RADIUS_M, SOLAR_IRRADIANCE,  # noqa: E402
                                                        SUN_ANGULAR_RADIUS_DEG, CameraView, batched_lut_jobs,
                                                        batched_lut_sets, frame_chain_cameras)
from planet_renderer_gb300.lighting import LightingState  # noqa: E402
from planet_renderer_gb300.ocean import OCEAN_SURFACE_ID, OceanConfig, OceanRenderer  # noqa: E402
from planet_renderer_gb300.postprocess import PostProcessor, PostprocessConfig  # noqa: E402
from planet_renderer_gb300.raster import TerrainRaster, synthetic_terrain  # noqa: E402
from planet_renderer_gb300.shading import OceanShading  # noqa: E402

R = EARTH_RADIUS_M
E = SOLAR_IRRADIANCE
SUN_DEG = SUN_ANGULAR_RADIUS_DEG
STARS = (4.0, 12.0)  # star contrast of the frame workloads
TF = camera.tangent_half_fov(60.0)
PRESETS = {"earth_baseline": (atm_config.earth_baseline, R), "earth_reference": (atm_config.earth_reference, R),
           "small_planet": (atm_config.small_planet, atm_config.SMALL_PLANET_RADIUS_M)}
AERIAL_NET, SKY_NET = (11, 4, 6), (10, 3, 3)  # inputs, hidden layers of 64, outputs


# ---- the cases ---------------------------------------------------------------
def listed() -> list[dict]:
    frame = {"kind": "frame", "preset": "earth_baseline", "layout": "wh", "channels": 3, "cameras": 3}
    return [
        # a preview thumbnail: launches and latency
        dict(frame, name="frame 96x54", width=96, height=54),
        # the frame chain of the benchmark: cameras at 2 km, 50 km and 2000 km
        dict(frame, name="frame 1920x1080", width=1920, height=1080),
        # a 4K frame loop over land and sea, the largest plain frame
        {"name": "fused 3840x2160", "kind": "fused", "preset": "earth_baseline", "layout": "wh", "channels": 3,
         "cameras": 2, "width": 3840, "height": 2160},
        # the same frame size with the learned composite
        {"name": "surrogate 3840x2160", "kind": "surrogate", "preset": "earth_baseline", "layout": "wh",
         "channels": 3, "cameras": 2, "width": 3840, "height": 2160},
        # the learned sky view, every pixel of a 4K image
        {"name": "sky net 3840x2160", "kind": "sky", "preset": "earth_baseline", "layout": "wh", "channels": 3,
         "mode": "net", "width": 3840, "height": 2160, "altitude_m": 2000.0},
        # an editor that changes an atmosphere parameter: all four LUTs at once
        {"name": "luts earth", "kind": "luts", "preset": "earth_baseline", "altitude_m": 2000.0},
        # time snapshots x cameras x parameter sets, uneven LUT sizes
        {"name": "batch 512", "kind": "batch", "snapshots": 16, "cameras": 8},
        # one optimiser step of an aerial network at the trainer's batch
        {"name": "train 16384", "kind": "train", "net": "aerial", "samples": 16384, "weighted": True},
        # the trainer's held-out evaluation
        {"name": "evaluate 65536", "kind": "evaluate", "net": "aerial", "samples": 65536},
        # the G-buffer of a 4K frame at the default patch budget
        {"name": "gbuffer 3840x2160", "kind": "gbuffer", "layout": "wh", "channels": 3, "rows": 16, "columns": 16,
         "resolution": 12, "altitude_m": 30.0, "width": 3840, "height": 2160},
        # the display transform of a 4K frame
        {"name": "post 3840x2160", "kind": "post", "layout": "wh", "channels": 3, "bloom": True, "tone_map": True,
         "passes": 4, "exposure_ev": 0.0, "width": 3840, "height": 2160},
        # a window of odd size, terrain patches to display, in one call after another
        {"name": "display 1366x767", "kind": "display", "layout": "wh", "channels": 3, "rows": 16, "columns": 16,
         "resolution": 12, "altitude_m": 30.0, "width": 1366, "height": 767},
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def _size(rng, tallest):
    height = int(_log(rng, 54, tallest))
    return min(int(height * rng.choice((4 / 3, 16 / 10, 16 / 9, 1.85))) + rng.randrange(3), tallest * 16 // 9), height


def draw(rng) -> dict:
    kind = rng.choice(("frame", "fused", "surrogate", "sky", "luts", "batch", "train", "evaluate", "gbuffer", "post",
                       "display"))
    c: dict = {"kind": kind}
    if kind in ("frame", "fused", "surrogate", "sky", "gbuffer", "post", "display"):
        c["width"], c["height"] = _size(rng, 1440 if kind in ("frame", "display") else 2160)
        # prepare_frame's lighting images have three channels
        c["layout"], c["channels"] = rng.choice(("wh", "hw")), 3 if kind == "frame" else rng.choice((3, 4))
    if kind in ("frame", "fused", "surrogate", "sky"):
        c["preset"] = rng.choice(("earth_baseline", "earth_reference"))
    if kind in ("frame", "fused", "surrogate"):
        c["cameras"] = rng.choice((2, 3)) if kind == "frame" else 2
    if kind in ("gbuffer", "display"):
        c["rows"], c["columns"], c["resolution"] = rng.randrange(4, 25), rng.randrange(4, 25), rng.choice((8, 12, 17, 24))
        c["altitude_m"] = _log(rng, 20.0, 2000.0)
    if kind == "sky":
        c["mode"], c["altitude_m"] = rng.choice(("net", "plain", "lut")), _log(rng, 10.0, 60_000.0)
    if kind == "luts":
        c["preset"], c["altitude_m"] = rng.choice(sorted(PRESETS)), _log(rng, 10.0, 2.0e6)
    if kind == "batch":
        c["snapshots"], c["cameras"] = rng.randrange(1, 17), rng.randrange(1, 9)
    if kind in ("train", "evaluate"):
        c["net"], c["samples"] = rng.choice(("aerial", "sky")), int(_log(rng, 256, 131072))
        if kind == "train":
            c["weighted"] = rng.random() < 0.5
    if kind == "post":
        c["bloom"], c["tone_map"], c["passes"] = rng.random() < 0.8, rng.random() < 0.8, rng.randrange(0, 9)
        c["exposure_ev"] = round(rng.uniform(-2.0, 2.0), 2)
    return c


# ---- inputs --------------------------------------------------------------------
def _generator(seed, salt=0):
    return torch.Generator(device="cuda").manual_seed((int(seed) * 1_000_003 + salt) % (1 << 62))


def _views(case, seed):
    """The cameras of a frame case; their suns follow the seed."""

    if case["kind"] == "sky":
        rng = np.random.default_rng(seed)
        return [CameraView(case["altitude_m"], float(rng.uniform(0.0, 80.0)), float(rng.uniform(0.0, 360.0)),
                           pitch_deg=8.0)]
    return frame_chain_cameras(seed)[:case["cameras"]]


def _light(view):
    return LightingState(view.sun_local, SUN_DEG, E)


def _as_layout(image, case):
    """(W, H, ...) images in the case's layout and channel count."""

    if image.dim() == 3 and image.shape[2] == 3 and case["channels"] == 4:
        image = torch.cat([image, torch.zeros_like(image[..., :1])], 2)
    return (image if case["layout"] == "wh" else image.transpose(0, 1)).contiguous()


def _rays(width, height, basis, tf):
    right, up, fwd = (torch.as_tensor(np.asarray(v, np.float64), device="cuda") for v in basis)
    sx = ((torch.arange(width, device="cuda", dtype=torch.float64) + 0.5) / width * 2.0 - 1.0) * (width / height)
    sy = (torch.arange(height, device="cuda", dtype=torch.float64) + 0.5) / height * 2.0 - 1.0
    d = right * sx[:, None, None] + up * sy[None, :, None] + fwd / tf
    return d / d.norm(dim=2, keepdim=True)


def _gbuffer(width, height, view, seed, salt):
    """A hilly planet seen by one camera, (W, H, ...): the ray's hit with a
    sphere displaced by a few octaves of waves; rays that miss are sky."""

    g = _generator(seed, salt)
    rays = _rays(width, height, view.basis, view.tangent_half_fov)
    amplitude = min(4000.0, 0.4 * view.altitude_m)
    k = torch.randn((6, 3), generator=g, device="cuda", dtype=torch.float64)
    k = k / k.norm(dim=1, keepdim=True) * (64.0 * 2.0 ** torch.arange(6, device="cuda"))[:, None]
    phase = torch.rand(6, generator=g, device="cuda", dtype=torch.float64) * 2.0 * math.pi
    o = R + view.altitude_m
    b = o * rays[..., 1]

    def relief(t):
        p = rays * t[..., None]
        p[..., 1] += o
        n = p / p.norm(dim=2, keepdim=True)
        return amplitude * sum(0.5 ** (j + 1) * torch.sin(n @ k[j] + phase[j]) for j in range(6)), n

    h = torch.zeros_like(b)
    for _ in range(4):
        disc = b * b - (o - R - h) * (o + R + h)
        t = -b - disc.clamp_min(0.0).sqrt()
        h, n = relief(t)
    hit = (disc > 0.0) & (t > 1.0)
    basis = torch.stack([torch.as_tensor(np.asarray(v, np.float64), device="cuda") for v in view.basis])
    position = torch.where(hit[..., None], (rays * t[..., None]) @ basis.T, 0.0).float()
    sun = torch.as_tensor(np.asarray(view.sun_local, np.float64), device="cuda")
    lit = (n @ sun).clamp_min(0.0)[..., None] + 0.05
    albedo = torch.tensor([0.16, 0.20, 0.12], device="cuda", dtype=torch.float64)
    e = torch.tensor(E, device="cuda", dtype=torch.float64)
    star = torch.rand((width, height), generator=g, device="cuda")
    star = torch.where(star < 0.01, 0.02 + 28.0 * star, 0.0)
    return {"position_view": position, "surface_id": torch.where(hit, 0, -1).int(),
            "scene_hdr": torch.where(hit[..., None], albedo * e / math.pi * lit, 0.0).float(),
            "space_hdr": torch.stack([star, star * 0.95, star * 1.05], 2), "relief": h.float(), "up": n.float()}


def _shading_images(gb):
    """The shading's G-buffer over land (relief above 0) and sea."""

    hit, h, n = gb["surface_id"] >= 0, gb["relief"], gb["up"]
    sea = hit & (h < 0.0)
    one = torch.ones_like(n)
    land = one * torch.tensor([0.16, 0.20, 0.12], device="cuda")
    return {"position": gb["position_view"], "normal": n,
            "albedo": torch.where(sea[..., None], one * torch.tensor([0.02, 0.05, 0.08], device="cuda"), land),
            "water_depth": torch.where(sea, -h, 0.0), "seabed_albedo": one * torch.tensor([0.30, 0.28, 0.20], device="cuda"),
            "seabed_normal": n, "slope_variance": torch.full_like(h, 0.01),
            "surface_id": torch.where(sea, OCEAN_SURFACE_ID, gb["surface_id"]).int(),
            "terrain_position": gb["position_view"], "terrain_normal": n, "terrain_albedo": land,
            "terrain_surface_id": torch.where(hit, 0, -1).int()}


def _network(shape, seed):
    """A network of trained-like weights: the output layer small, its bias the
    log of an ordinary radiance."""

    net = Mlp(*shape, seed=seed % (1 << 31))
    p = net.params()
    n_in, _, n_out = shape
    p[-(HIDDEN + 1) * n_out:-n_out] *= 0.25
    p[-n_out:] = -2.5
    net.set_params(p)
    return net


def _train_set(shape, n, seed, weighted):
    g = _generator(seed, 7)
    n_in, _, n_out = shape
    x = torch.rand((n, n_in), generator=g, device="cuda") * 2.0 - 1.0
    y = torch.randn((n, n_out), generator=g, device="cuda")  # standardised targets
    w = torch.rand((n, n_out), generator=g, device="cuda") * 2.0 if weighted else None
    return x, y, w


def _shape(case):
    return AERIAL_NET if case["net"] == "aerial" else SKY_NET


def _terrain(case, seed):
    """A mesh frame's patches over a coast and the camera above it."""

    mesh = synthetic_terrain(case["width"], case["height"], TF, altitude_m=case["altitude_m"], pitch_degrees=6.0,
                             rows=case["rows"], columns=case["columns"], resolution=case["resolution"],
                             relief_m=200.0, base_height_m=0.0, rise_m_per_km=10.0, seed=int(seed) % (1 << 31))
    mesh["skirt_mask"].zero_()  # every seam of these patches is closed: no skirt is drawn
    return mesh


def _mesh_state(case, seed):
    mesh = _terrain(case, seed)
    raster = TerrainRaster(case["width"], case["height"], int(mesh["view"].shape[0]), int(mesh["triangles"].shape[0]),
                           layout=case["layout"])
    return {"mesh": mesh, "raster": raster,
            "gbuffer": raster.allocate_gbuffer(case["channels"], snapshot=True, ocean=True),
            "sea": OceanRenderer(case["width"], case["height"], OceanConfig(), layout=case["layout"]),
            "planet": (np.array([1.0, 0.0, 0.0]), np.array([0.0, 1.0, 0.0]), np.array([0.0, 0.0, 1.0])),
            "time": float(np.random.default_rng(seed).uniform(0.0, 600.0))}


def _blank(case):
    shape = (case["width"], case["height"]) if case["layout"] == "wh" else (case["height"], case["width"])
    return torch.zeros(shape + (case["channels"],), device="cuda")


def _renderer(case):
    make, radius = PRESETS[case.get("preset", "earth_baseline")]
    return AtmosphereRenderer(case.get("width", 16), case.get("height", 16), make(), layout=case.get("layout", "wh")), radius


def _batch_jobs(case, seed):
    """The batched workload's jobs: sizes by the case alone, suns and cameras by the seed."""

    sized = batched_lut_jobs(2027, case["snapshots"], case["cameras"])
    return [dataclasses.replace(j, width=k.width, height=k.height, depth=k.depth)
            for j, k in zip(batched_lut_jobs(seed, case["snapshots"], case["cameras"]), sized)]


def _hdr_image(case, seed):
    """An HDR frame: smooth radiance, speckle and a few highlights above the bloom threshold."""

    g = _generator(seed, 3)
    w, h = case["width"], case["height"]
    x = torch.linspace(0.0, 6.0, w, device="cuda")[:, None, None]
    y = torch.linspace(0.0, 4.0, h, device="cuda")[None, :, None]
    tint = torch.rand(3, generator=g, device="cuda") + 0.3
    v = tint * (0.4 + 0.35 * torch.sin(x + tint) * torch.cos(y)) + 0.02 * torch.rand((w, h, 3), generator=g, device="cuda")
    spot = torch.rand((w, h, 1), generator=g, device="cuda")
    return torch.where(spot < 0.002, v + 5000.0 * spot, v)


def prepare(case, seed):
    kind = case["kind"]
    s: dict = {"case": case, "kind": kind}
    if kind in ("frame", "fused", "surrogate", "sky"):
        s["renderer"], _ = _renderer(case)
        s["views"] = []
        for k, v in enumerate(_views(case, seed)):
            view = {"view": v, "radius": v.camera_radius_m, "sun": tuple(float(c) for c in v.sun_local),
                    "disk": _light(v).sun_disk_radiance, "basis": v.basis, "tf": v.tangent_half_fov,
                    "hdr": _blank(case)}
            if kind != "sky":
                gb = _gbuffer(case["width"], case["height"], v, seed, k)
                images = _shading_images(gb) if kind == "fused" else {}
                view["space"] = _as_layout(gb["space_hdr"], case)
                view["images"] = {n: _as_layout(t, case) for n, t in images.items()}
                if kind != "fused":
                    view.update(scene=_as_layout(gb["scene_hdr"], case), sid=_as_layout(gb["surface_id"], case),
                                position=_as_layout(gb["position_view"], case))
            s["views"].append(view)
        if kind in ("surrogate", "sky"):
            s["surrogate"] = Surrogate(_network(AERIAL_NET, seed + 1) if kind == "surrogate" else None,
                                       _network(SKY_NET, seed + 2),
                                       aerial_above_shell=_network(AERIAL_NET, seed + 3) if kind == "surrogate" else None)
        v = s["views"][0]
        s["renderer"].update(R, v["radius"], v["sun"], E, SUN_DEG)
    elif kind == "luts":
        s["renderer"], s["radius"] = _renderer(case)
        v = frame_chain_cameras(seed)[0]
        sun = v.sun_local
        s["args"] = {"planet_radius_m": s["radius"], "camera_altitude_m": case["altitude_m"],
                     "sun_zenith_cosine": float(np.float32(sun[1])), "sun_local": tuple(float(c) for c in sun),
                     "view_basis": v.basis, "tangent_half_fov": TF}
    elif kind == "batch":
        s["builder"] = BatchedLutBuilder(batched_lut_sets())
        s["jobs"] = _batch_jobs(case, seed)
        s["prepared"] = s["builder"].prepare(s["jobs"])
        s["arena"] = torch.empty((s["prepared"][1], 4), device="cuda")
    elif kind == "train":
        s["net"] = Mlp(*_shape(case), seed=seed % (1 << 31))
        s["data"] = _train_set(_shape(case), case["samples"], seed, case["weighted"])
    elif kind == "evaluate":
        s["net"] = _network(_shape(case), seed)
        s["net"].pack()
        s["x"] = _train_set(_shape(case), case["samples"], seed, False)[0]
    elif kind == "gbuffer":
        s.update(_mesh_state(case, seed))
    elif kind == "post":
        s["post"] = PostProcessor(case["width"], case["height"], PostprocessConfig(bloom_passes=case["passes"]),
                                  layout=case["layout"])
        s["hdr"] = _as_layout(_hdr_image(case, seed), case)
        s["display"] = torch.zeros_like(s["hdr"])
    elif kind == "display":
        s.update(_mesh_state(case, seed))
        s["renderer"], _ = _renderer(case)
        s["post"] = PostProcessor(case["width"], case["height"], PostprocessConfig(), layout=case["layout"])
        rng = np.random.default_rng(seed)
        sun = camera.sun_local(float(rng.uniform(0.0, 360.0)), float(rng.uniform(5.0, 60.0)))
        s["sun"] = tuple(float(c) for c in sun)
        s["disk"] = LightingState(sun, SUN_DEG, E).sun_disk_radiance
        s["space"], s["hdr"], s["display"] = _blank(case), _blank(case), _blank(case)
        s["altitudes"], s["pass"] = (case["altitude_m"], case["altitude_m"] + 0.5), 0
    else:
        raise ValueError(f"unknown kind {kind}")
    return s


# ---- one pass -------------------------------------------------------------------
def _produce_gbuffer(s):
    c, g = s["case"], s["gbuffer"]
    s["raster"].render(s["mesh"], 0.5, TF, g)
    s["sea"].rasterize_gbuffer(g, R, c["altitude_m"], s["planet"], s["mesh"]["view_basis"], TF, s["time"], 0)


def run(s):
    kind = s["kind"]
    if kind == "frame":
        r = s["renderer"]
        for v in s["views"]:
            r.update(R, v["radius"], v["sun"], E, SUN_DEG)
            r.prepare_frame(v["position"], v["sid"], R, v["radius"], v["sun"], E, SUN_DEG, v["basis"], v["tf"])
            r.composite(v["scene"], v["space"], v["sid"], v["position"], v["hdr"], R, v["radius"], v["sun"], E,
                        v["disk"], SUN_DEG, v["basis"], v["tf"], *STARS)
        # the renderer's lighting images are the last camera's
        return {"hdr": [v["hdr"] for v in s["views"]], "sun_t": r.surface_sun_transmittance,
                "sky_l": r.surface_sky_radiance}
    if kind == "fused":
        r = s["renderer"]
        for v in s["views"]:
            r.update(R, v["radius"], v["sun"], E, SUN_DEG)
            r.render_frame(v["images"], v["space"], v["hdr"], R, v["radius"], v["sun"], E, v["disk"], SUN_DEG,
                           v["basis"], v["tf"], *STARS, ocean=OceanShading())
        return [v["hdr"] for v in s["views"]]
    if kind == "surrogate":
        r = s["renderer"]
        for v in s["views"]:
            r.update(R, v["radius"], v["sun"], E, SUN_DEG)
            r.composite_surrogate(v["scene"], v["space"], v["sid"], v["position"], v["hdr"], R, v["radius"], v["sun"],
                                  E, v["disk"], SUN_DEG, v["basis"], v["tf"], *STARS, surrogate=s["surrogate"])
        return [v["hdr"] for v in s["views"]]
    if kind == "sky":
        v = s["views"][0]
        s["renderer"].sky_pixels(v["hdr"], R, v["radius"], v["sun"], E, SUN_DEG, v["basis"], v["tf"],
                                 mode=s["case"]["mode"], surrogate=s["surrogate"])
        return v["hdr"]
    if kind == "luts":
        r = s["renderer"]
        out = []
        for name, field in (("transmittance", r.transmittance_lut), ("multi_scattering", r.multi_scattering_lut),
                            ("sky_view", r.sky_view_lut), ("aerial", r.aerial_scattering_lut)):
            r.build_lut(name, **s["args"])
            out.append(field.to_torch())
        return out
    if kind == "batch":
        return s["builder"].build(s["jobs"], arena=s["arena"], prepared=s["prepared"]).arena
    if kind == "train":
        x, y, w = s["data"]
        loss = s["net"].train_step(x, y, weights=w)
        return {"loss": loss, "params": s["net"].params()}
    if kind == "evaluate":
        return {"f32": s["net"].forward(s["x"], "f32"), "bf16": s["net"].forward(s["x"], "bf16")}
    if kind == "gbuffer":
        _produce_gbuffer(s)
        return s["gbuffer"]
    if kind == "post":
        c = s["case"]
        s["post"].process(s["hdr"], s["display"], c["exposure_ev"], bloom=c["bloom"], tone_map=c["tone_map"])
        return s["display"]
    # display: the camera bobs between two heights, so that its sky-view LUT is rebuilt every frame
    _produce_gbuffer(s)
    radius = R + s["altitudes"][s["pass"] & 1]
    s["pass"] += 1
    r, basis = s["renderer"], s["mesh"]["view_basis"]
    r.update(R, radius, s["sun"], E, SUN_DEG)
    r.render_frame(s["gbuffer"], s["space"], s["hdr"], R, radius, s["sun"], E, s["disk"], SUN_DEG, basis, TF, *STARS,
                   ocean=OceanShading())
    s["post"].process(s["hdr"], s["display"], 0.0, bloom=True, tone_map=True)
    return {"hdr": s["hdr"], "display": s["display"]}


# ---- what a pass cannot do without ------------------------------------------------
SAMPLE_FLOPS = 406.0  # of one constant-source segment, counted on the reference's algorithm
SAMPLES_PER_PIXEL = 36.0  # of a composite, over the frame cameras (sky pixels take none)


def _mlp_flops(shape):
    return 2.0 * sum(o * i for o, i in layer_shapes(*shape))


def work(case) -> dict:
    kind = case["kind"]
    px = float(case.get("width", 0) * case.get("height", 0))
    rgb = 4.0 * case.get("channels", 3)
    if kind in ("frame", "fused", "surrogate"):
        cfg, n = PRESETS[case["preset"]][0](), case["cameras"]
        sky = cfg.sky_view_lut_width * cfg.sky_view_lut_height * cfg.sky_view_steps * 309.0
        # position, scene, space, id in; hdr out; lighting images out (frame); shading images in (fused)
        per_px = 4 * rgb + 4.0 + {"frame": 2 * rgb, "fused": 6 * rgb + 12.0, "surrogate": 0.0}[kind]
        flops = _mlp_flops(AERIAL_NET) if kind == "surrogate" else SAMPLES_PER_PIXEL * SAMPLE_FLOPS
        return {"bytes": n * px * per_px, "flops": n * (px * flops + sky)}
    if kind == "sky":
        cfg = PRESETS[case["preset"]][0]()
        flops = {"net": _mlp_flops(SKY_NET), "plain": cfg.sky_view_steps * 309.0, "lut": 60.0}[case["mode"]]
        return {"bytes": px * rgb, "flops": px * flops}
    if kind == "luts":
        c = PRESETS[case["preset"]][0]()
        t, m = c.transmittance_lut_width * c.transmittance_lut_height, c.multi_scattering_lut_width * c.multi_scattering_lut_height
        s, a = c.sky_view_lut_width * c.sky_view_lut_height, c.aerial_lut_width * c.aerial_lut_height * c.aerial_lut_depth
        return {"bytes": 12.0 * (t + m + s + a),
                "flops": (72.0 * t * c.transmittance_steps + 266.0 * m * c.multi_scattering_directions * c.multi_scattering_steps
                          + 309.0 * s * c.sky_view_steps + 302.0 * a * c.aerial_steps_per_slice)}
    if kind == "batch":
        jobs, sets = _batch_jobs(case, 1), batched_lut_sets()
        return {"bytes": 16.0 * sum(j.texels for j in jobs),
                "flops": 305.0 * sum(j.samples(sets[j.param_set][0]) for j in jobs)}
    if kind in ("train", "evaluate"):
        shape, n = _shape(case), float(case["samples"])
        n_params = sum(o * i + o for o, i in layer_shapes(*shape))
        if kind == "train":  # samples, parameters and both Adam moments
            return {"bytes": 4.0 * (n * (shape[0] + shape[2] * (2 if case["weighted"] else 1)) + 6 * n_params),
                    "flops": 3.0 * n * _mlp_flops(shape)}
        return {"bytes": 2 * 4.0 * (n * (shape[0] + shape[2]) + n_params), "flops": 2.0 * n * _mlp_flops(shape)}
    if kind == "post":
        return {"bytes": 2 * px * rgb, "flops": px * 150.0}
    # the G-buffer and its terrain snapshot written once, the patches read once; a wave solve per sea pixel
    verts = case["rows"] * case["columns"] * ((case["resolution"] + 1) ** 2 + 4 * (case["resolution"] + 1))
    gbuffer = {"bytes": px * (8 * rgb + 44.0) + verts * 48.0, "flops": px * 900.0}
    if kind == "gbuffer":
        return gbuffer
    return {"bytes": gbuffer["bytes"] + px * (8 * rgb + 16.0) + 2 * px * rgb,
            "flops": gbuffer["flops"] + px * (SAMPLES_PER_PIXEL * SAMPLE_FLOPS + 150.0)}


# ---- the same in 64 bits -------------------------------------------------------------
def _f32(v):
    """Arguments as the entry points take them: rounded to float32."""

    return torch.as_tensor(np.asarray(v, np.float64).astype(np.float32).astype(np.float64), device="cuda")


def _dot(a, b):
    return (a * b).sum(-1)


def _unit(v):
    return v / v.norm(dim=-1, keepdim=True)


class Atmosphere64:
    """The reference's atmosphere in float64 torch: scalars per ray as (n,)
    tensors, colours as (n, 3)."""

    def __init__(self, config, radius):
        self.c, self.R, self.top = config, float(radius), float(np.float32(config.top_altitude_m))
        self.ar = float(np.float32(math.radians(SUN_DEG)))
        self.E = _f32(E)
        k = lambda name: _f32(getattr(config, name))  # noqa: E731
        self.br, self.ms, self.me, self.bo = (k("rayleigh_scattering_per_m"), k("mie_scattering_per_m"),
                                              k("mie_extinction_per_m"), k("absorption_extinction_per_m"))
        self.albedo = k("ground_albedo")
        self.rho_top = self.rho(torch.tensor(self.top, dtype=torch.float64, device="cuda"))
        self.t = self._transmittance()
        self.m = self._multi_scattering()

    # geometry
    def rho(self, h):
        h = h.clamp_min(0.0)
        return (h * (2.0 * self.R + h)).sqrt()

    def altitude(self, h0, cosv, t):
        d = h0 * (2.0 * self.R + h0) + 2.0 * (self.R + h0) * cosv * t + t * t
        return d / ((self.R * self.R + d).clamp_min(0.0).sqrt() + self.R)

    def roots(self, h0, cosv, shell):
        b = (self.R + h0) * cosv
        c = (h0 - shell) * (2.0 * self.R + h0 + shell)
        disc = b * b - c
        q = -b - torch.where(b < 0.0, -1.0, 1.0) * disc.clamp_min(0.0).sqrt()
        other = torch.where(q.abs() > 1e-12, c / q, q)
        hit = disc >= 0.0
        return torch.where(hit, torch.minimum(q, other), 1e30), torch.where(hit, torch.maximum(q, other), -1e30), hit

    def segment(self, h0, cosv, eps=1e-3):
        near, far, hit = self.roots(h0, cosv, self.top)
        start, end = near.clamp_min(0.0), far
        valid = hit & (end > start)
        gn, gf, gh = self.roots(h0, cosv, 0.0)
        g = torch.where(gn > start + eps, gn, torch.where(gf > start + eps, gf, 1e30))
        ground = valid & gh & (g < end)
        return start, torch.where(ground, g, end), valid, ground

    @staticmethod
    def warp(closest, start, end, f):
        c = torch.minimum(torch.maximum(closest, start), end)
        eps = ((end - start) * 1e-6).clamp_min(1e-5)
        first, last = start + (end - start) * f * f, end - (end - start) * (1.0 - f) ** 2
        mid = c - (c - start) * (1.0 - 2.0 * f) ** 2 if f < 0.5 else c + (end - c) * (2.0 * f - 1.0) ** 2
        return torch.where(c <= start + eps, first, torch.where(c >= end - eps, last, mid))

    # medium
    def density(self, h):
        inside = (h >= 0.0) & (h <= self.top)
        c = self.c
        return (torch.where(inside, (-h / c.rayleigh_scale_height_m).exp(), 0.0),
                torch.where(inside, (-h / c.mie_scale_height_m).exp(), 0.0),
                torch.where(inside, (1.0 - (h - c.absorption_peak_altitude_m).abs() / c.absorption_half_width_m).clamp_min(0.0), 0.0))

    def extinction(self, d):
        return d[0][:, None] * self.br + d[1][:, None] * self.me + d[2][:, None] * self.bo

    def phases(self, c):
        g = self.c.mie_phase_g
        c = c.clamp(-1.0, 1.0)
        ray = 3.0 * (1.0 + c * c) / (16.0 * math.pi)
        mie = 3.0 * (1.0 - g * g) * (1.0 + c * c) / (8.0 * math.pi * (2.0 + g * g) * (1.0 + g * g - 2.0 * g * c).clamp_min(1e-8) ** 1.5)
        return ray, mie

    # LUTs, (H, W, 3)
    @staticmethod
    def tap(lut, u, v):
        h, w, _ = lut.shape
        x, y = (u * w - 0.5).clamp(0.0, w - 1), (v * h - 0.5).clamp(0.0, h - 1)
        x0, y0 = x.floor().long(), y.floor().long()
        x1, y1 = (x0 + 1).clamp_max(w - 1), (y0 + 1).clamp_max(h - 1)
        fx, fy = (x - x0)[:, None], (y - y0)[:, None]
        return ((lut[y0, x0] * (1 - fx) + lut[y0, x1] * fx) * (1 - fy) + (lut[y1, x0] * (1 - fx) + lut[y1, x1] * fx) * fy)

    @staticmethod
    def grid(w, h):
        y, x = torch.meshgrid(torch.arange(h, device="cuda"), torch.arange(w, device="cuda"), indexing="ij")
        return ((x.reshape(-1).double() + 0.5) / w), ((y.reshape(-1).double() + 0.5) / h)

    def _transmittance(self):
        c = self.c
        u, v = self.grid(c.transmittance_lut_width, c.transmittance_lut_height)
        rho = self.rho_top * v
        h = rho * rho / ((rho * rho + self.R ** 2).sqrt() + self.R)
        dmin = self.top - h
        dist = dmin + u * (rho + self.rho_top - dmin)
        cosv = (((self.top - h) * (2.0 * self.R + self.top + h) - dist * dist) / (2.0 * (self.R + h) * dist)).clamp(-1.0, 1.0)
        closest, zero, n = -(self.R + h) * cosv, torch.zeros_like(h), c.transmittance_steps
        od, d0 = torch.zeros((h.numel(), 3), dtype=torch.float64, device="cuda"), zero
        for i in range(n):
            d1 = self.warp(closest, zero, dist, (i + 1) / n)
            od = od + self.extinction(self.density(self.altitude(h, cosv, 0.5 * (d0 + d1)))) * (d1 - d0)[:, None]
            d0 = d1
        return (-od.clamp_max(80.0)).exp().reshape(c.transmittance_lut_height, c.transmittance_lut_width, 3)

    def sample_t(self, h, cosv):
        h = h.clamp(0.0, self.top)
        rho, r = self.rho(h), self.R + h
        d = (-r * cosv + (r * r * cosv * cosv + (self.top - h) * (2.0 * self.R + self.top + h)).clamp_min(0.0).sqrt()).clamp_min(0.0)
        dmin = self.top - h
        u = ((d - dmin) / (rho + self.rho_top - dmin).clamp_min(1e-6)).clamp(0.0, 1.0)
        return self.tap(self.t, u, (rho / self.rho_top).clamp(0.0, 1.0))

    def horizon(self, h):
        return -self.rho(h) / (self.R + h.clamp_min(0.0))

    def solar(self, h, sc):
        """Sun transmittance of the finite disk, and the disk's visible share."""

        hz, sz = self.horizon(h).clamp(-1.0, 1.0).acos(), sc.clamp(-1.0, 1.0).acos()
        n = ((hz - sz) / self.ar).clamp(-1.0, 1.0)
        vis = ((-n).acos() + n * (1.0 - n * n).clamp_min(0.0).sqrt()) / math.pi
        rz = torch.minimum(sz, hz - 0.25 * self.ar).clamp_min(0.0)
        return self.sample_t(h, rz.cos()) * vis[:, None], vis

    def sample_ms(self, h, sc):
        hc = self.horizon(h)
        low = 0.5 * (1.0 - ((hc - sc) / (hc + 1.0).clamp_min(1e-6)).clamp(0.0, 1.0).sqrt())
        high = 0.5 + 0.5 * ((sc - hc) / (1.0 - hc).clamp_min(1e-6)).clamp(0.0, 1.0).sqrt()
        return self.tap(self.m, torch.where(sc < hc, low, high), (h / self.top).clamp(0.0, 1.0).sqrt())

    @staticmethod
    def integral(ext, step):
        x = (ext * step[:, None]).clamp_max(80.0)
        return (-x).exp(), torch.where(ext > 1e-14, -torch.expm1(-x) / ext.clamp_min(1e-14), step[:, None])

    def _multi_scattering(self):
        c = self.c
        u, v = self.grid(c.multi_scattering_lut_width, c.multi_scattering_lut_height)
        nd, n = c.multi_scattering_directions, c.multi_scattering_steps
        h0 = v * v * self.top
        hc = self.horizon(h0)
        sc = torch.where(u < 0.5, hc - (hc + 1.0) * (1.0 - 2.0 * u) ** 2, hc + (1.0 - hc) * (2.0 * u - 1.0) ** 2).clamp(-1.0, 1.0)
        k = torch.arange(nd, device="cuda", dtype=torch.float64)
        dc, az = 1.0 - 2.0 * (k + 0.5) / nd, k * 2.39996323
        ds = (1.0 - dc * dc).clamp_min(0.0).sqrt()
        texels = h0.numel()
        h0, sc = h0.repeat_interleave(nd), sc.repeat_interleave(nd)
        ray = torch.stack([ds * az.cos(), dc, ds * az.sin()], 1).repeat(texels, 1)
        sun = torch.stack([(1.0 - sc * sc).clamp_min(0.0).sqrt(), sc, torch.zeros_like(sc)], 1)
        start, end, valid, ground = self.segment(h0, ray[:, 1], max(0.001, self.R * 1e-8))
        end = torch.where(valid, end, start)
        pr, pm = self.phases(_dot(ray, sun))
        closest = -(self.R + h0) * ray[:, 1]
        L = torch.zeros((h0.numel(), 3), dtype=torch.float64, device="cuda")
        F, T = torch.zeros_like(L), torch.ones_like(L)

        def sun_cosine(t):
            return (_dot(ray, sun) * t + (self.R + h0) * sc) / (self.R + self.altitude(h0, ray[:, 1], t))

        d0 = start
        for i in range(n):
            d1 = self.warp(closest, start, end, (i + 1) / n)
            t = 0.5 * (d0 + d1)
            h = self.altitude(h0, ray[:, 1], t)
            d = self.density(h)
            sT, sI = self.integral(self.extinction(d), d1 - d0)
            st, _ = self.solar(h, sun_cosine(t))
            L = L + T * self.E * st * ((d[0] * pr)[:, None] * self.br + (d[1] * pm)[:, None] * self.ms) * sI
            F = F + T * (d[0][:, None] * self.br + d[1][:, None] * self.ms) * sI
            T, d0 = T * sT, d1
        gsc = sun_cosine(end)
        gt, _ = self.solar(torch.zeros_like(gsc), gsc)
        L = L + torch.where(ground[:, None], T * self.albedo * self.E * gt * gsc.clamp_min(0.0)[:, None] / math.pi, 0.0)
        L, F = (torch.where(valid[:, None], a, 0.0).reshape(texels, nd, 3).mean(1) for a in (L, F))
        return (L / (1.0 - F.clamp(0.0, 0.95))).clamp_min(0.0).reshape(c.multi_scattering_lut_height, c.multi_scattering_lut_width, 3)

    # the march
    def ray(self, h0, d, sun):
        """What the samples of rays d (n, 3) from altitudes h0 (n,) share; sun (n, 3)."""

        rs = _dot(d, sun)
        pr, pm = self.phases(rs)
        return {"h0": h0, "cosv": d[:, 1], "rs": rs, "s0": (self.R + h0) * sun[:, 1], "ER": self.E * self.br * pr[:, None],
                "EM": self.E * self.ms * pm[:, None], "closest": -(self.R + h0) * d[:, 1]}

    def source(self, q, d0, d1):
        t = 0.5 * (d0 + d1)
        h = self.altitude(q["h0"], q["cosv"], t)
        d = self.density(h)
        T, I = self.integral(self.extinction(d), (d1 - d0).clamp_min(0.0))
        sc = (q["s0"] + t * q["rs"]) / (self.R + h)
        st, vis = self.solar(h, sc)
        src = st * (q["ER"] * d[0][:, None] + q["EM"] * d[1][:, None])
        src = src + (d[0][:, None] * self.br + d[1][:, None] * self.ms) * self.sample_ms(h, sc)
        return src * I, T, vis

    def march(self, q, start, end, n):
        L, T = torch.zeros_like(q["ER"]), torch.ones_like(q["ER"])
        d0 = start
        for i in range(n):
            d1 = self.warp(q["closest"], start, end, (i + 1) / n)
            l, t, _ = self.source(q, d0, d1)
            L, T, d0 = L + T * l, T * t, d1
        return L, T

    def sky_rays(self, h0, d, sun):
        out = []
        for a in range(0, h0.numel(), 1 << 20):
            p = slice(a, a + (1 << 20))
            start, end, valid, _ = self.segment(h0[p], d[p, 1])
            L, _ = self.march(self.ray(h0[p], d[p], sun[p]), start, torch.where(valid, end, start), self.c.sky_view_steps)
            out.append(torch.where(valid[:, None], L, 0.0).clamp_min(0.0))
        return torch.cat(out)

    def sky_texels(self, w, h, altitude, sun_cos):
        """Camera altitude, ray and sun of every texel of a sky-view LUT, in [y][x] order."""

        u, v = self.grid(w, h)
        alt = torch.full_like(u, float(np.float32(max(altitude, 0.0))))
        hz = math.pi - (self.rho(alt) / (self.R + alt)).clamp(0.0, 1.0).acos()
        zen = torch.where(v < 0.5, hz * (1.0 - (1.0 - 2.0 * v) ** 2), hz + (math.pi - hz) * (2.0 * v - 1.0) ** 2)
        az = u * math.pi
        d = torch.stack([zen.sin() * az.cos(), zen.cos(), zen.sin() * az.sin()], 1)
        sun = torch.tensor([[math.sqrt(max(1.0 - sun_cos * sun_cos, 0.0)), sun_cos, 0.0]], dtype=torch.float64, device="cuda")
        return alt, d, sun.expand_as(d)

    def sky_view(self, w, h, altitude, sun_cos):
        return self.sky_rays(*self.sky_texels(w, h, altitude, sun_cos)).reshape(h, w, 3)

    def columns(self, w, h, frame, altitude, sun, basis, tf):
        """Camera altitude, ray and sun of every column of an aerial volume, in [y][x] order."""

        u, v = self.grid(w, h)
        b = _f32(basis)
        aspect, tf = float(np.float32(frame[0] / frame[1])), float(np.float32(tf))
        d = _unit(((u * 2.0 - 1.0) * aspect)[:, None] * b[0] + (v * 2.0 - 1.0)[:, None] * b[1] + b[2] / tf)
        return torch.full_like(u, float(np.float32(max(altitude, 0.0)))), d, _f32(sun).expand_as(d)

    def slices(self, alt, d, sun, depth):
        """Cumulative in-scattering at the depth slices of columns, (D, n, 3)."""

        q = self.ray(alt, d, sun)
        start, end, valid, ground = self.segment(alt, d[:, 1])
        cut = valid & ~ground & (q["closest"] > start) & (q["closest"] < end)
        start = torch.where(valid, start, 0.0)
        end = torch.where(valid, torch.where(cut, q["closest"], end), 0.0)
        L, T, out, n = torch.zeros_like(d), torch.ones_like(d), [], self.c.aerial_steps_per_slice
        for k in range(depth):
            a = start + (end - start) * (max(k - 1, 0) / (depth - 1))
            e = start + (end - start) * (k / (depth - 1))
            d0 = a
            for i in range(n if k else 0):
                d1 = self.warp(q["closest"], a, e, (i + 1) / n)
                l, t, _ = self.source(q, d0, d1)
                L, T, d0 = L + T * l, T * t, d1
            out.append(L.clamp_min(0.0))
        return torch.stack(out)

    # a frame's pixels
    def lighting(self, altitude, basis, sun, position):
        p = position.double() @ _f32(basis)
        t = p.norm(dim=1)
        d = p / t.clamp_min(1.0)[:, None]
        alt = torch.full_like(t, altitude)
        h = self.altitude(alt, d[:, 1], t)
        sc = ((self.R + altitude) * sun[1] + t * (d @ sun)) / (self.R + h)
        st, _ = self.solar(h, sc)
        return st, self.sample_ms(h, sc).clamp_min(0.0)

    def shadow_roots(self, o_y, d, sun):
        o = torch.zeros_like(d)
        o[:, 1] = o_y
        op, rp = o - sun * (o @ sun)[:, None], d - sun * (d @ sun)[:, None]
        quad, hl, pl = _dot(rp, rp), _dot(op, rp), op.norm(dim=1)
        disc = hl * hl - quad * (pl - self.R) * (pl + self.R)
        ok = (quad > 1e-8) & (disc >= 0.0)
        root = disc.clamp_min(0.0).sqrt()
        ts = [(-hl + s * root) / quad.clamp_min(1e-8) for s in (-1.0, 1.0)]
        return [(t, ok & (((o + d * t[:, None]) @ sun) < 0.0)) for t in ts]

    def surface(self, altitude, d, sun, distance):
        """In-scattering and transmittance between the camera and a surface."""

        n, sub = self.c.aerial_horizon_raymarch_steps, self.c.aerial_terminator_substeps
        alt = torch.full_like(distance, altitude)
        near, far, hit = self.roots(alt, d[:, 1], self.top)
        start, end = near.clamp_min(0.0), torch.minimum(distance, far)
        valid = hit & (end > start)
        start = torch.where(valid, start, 0.0)
        end = torch.where(valid, end, start)
        q = self.ray(alt, d, sun.expand_as(d))
        shadow = self.shadow_roots(self.R + altitude, d, sun)
        L, T = torch.zeros_like(d), torch.ones_like(d)
        d0 = start
        for i in range(n):
            d1 = self.warp(q["closest"], start, end, (i + 1) / n)
            l, t, vis = self.source(q, d0, d1)
            mid, width = 0.5 * (d0 + d1), (d1 - d0).clamp_min(1e-4)
            near_root = torch.full_like(mid, 1e30)
            for root, ok in shadow:
                near_root = torch.where(ok, torch.minimum(near_root, (mid - root).abs()), near_root)
            prox = (2.0 - near_root / width).clamp(0.0, 1.0)
            weight = torch.maximum(prox * prox * (3.0 - 2.0 * prox), 4.0 * vis * (1.0 - vis))
            at = (weight > 0.0).nonzero()[:, 0]
            if at.numel():
                sq, a, b = {k: x[at] for k, x in q.items()}, d0[at], d1[at]
                fl, ft = torch.zeros_like(l[at]), torch.ones_like(l[at])
                for k in range(sub):
                    x, y, _ = self.source(sq, a + (b - a) * (k / sub), a + (b - a) * ((k + 1) / sub))
                    fl, ft = fl + ft * x, ft * y
                w = weight[at][:, None]
                l[at], t[at] = l[at] * (1.0 - w) + fl * w, t[at] * (1.0 - w) + ft * w
            L, T, d0 = L + T * l, T * t, d1
        taps = []
        for x in (end, start):
            h = self.altitude(alt, d[:, 1], x)
            taps.append(self.sample_t(h, -(x - q["closest"]) / (self.R + h)))
        ratio = (taps[0] / taps[1].clamp_min(1e-6)).clamp(0.0, 1.0)
        return torch.where(valid[:, None], L.clamp_min(0.0), 0.0), torch.where(valid[:, None], ratio, 1.0)

    def sky_tap(self, lut, altitude, d, sun):
        alt = torch.full_like(d[:, 1], altitude)
        hz = math.pi - (self.rho(alt) / (self.R + alt)).clamp(0.0, 1.0).acos()
        zen = d[:, 1].clamp(-1.0, 1.0).acos()
        vl, sl = (d[:, 0] ** 2 + d[:, 2] ** 2).sqrt(), (sun[0] ** 2 + sun[2] ** 2).sqrt()
        ra = torch.where((vl > 1e-6) & (sl > 1e-6),
                         ((d[:, 0] * sun[0] + d[:, 2] * sun[2]) / (vl * sl).clamp_min(1e-12)).clamp(-1.0, 1.0).acos(), 0.0)
        low = 0.5 * (1.0 - (1.0 - (zen / hz).clamp(0.0, 1.0)).sqrt())
        high = 0.5 + 0.5 * ((zen - hz) / (math.pi - hz).clamp_min(1e-6)).clamp(0.0, 1.0).sqrt()
        return self.tap(lut, ra / math.pi, torch.where(zen < hz, low, high))

    def sky_pixel(self, lut, altitude, d, sun, color, space, disk, tf, height):
        alt = torch.full_like(d[:, 1], altitude)
        start, _, valid, ground = self.segment(alt, d[:, 1])
        h = self.altitude(alt, d[:, 1], start)
        tr = self.sample_t(h, (start + (self.R + alt) * d[:, 1]) / (self.R + h))
        tr = torch.where(valid[:, None], torch.where(ground[:, None], 0.0, tr), 1.0)
        sky = self.sky_tap(lut, altitude, d, sun)
        star = space * tr
        lw = torch.tensor([0.2126, 0.7152, 0.0722], dtype=torch.float64, device="cuda")
        vis = (((star @ lw) / (sky @ lw).clamp_min(1e-5) - STARS[0]) / (STARS[1] - STARS[0])).clamp(0.0, 1.0)
        vis = (vis * vis * (3.0 - 2.0 * vis))[:, None]
        pf = math.atan2(tf * 1.41421356 / height, 1.0)
        cov = ((self.ar + pf - (d @ sun).clamp(-1.0, 1.0).acos()) / (2.0 * pf)).clamp(0.0, 1.0)
        cov = (cov * cov * (3.0 - 2.0 * cov))[:, None]
        return sky + color * tr + star * vis + _f32(disk) * tr * cov

    def composite(self, v, scene, space, sid, position, width, height):
        """The COMPOSITE view of (W, H, 3) images, flattened to (W * H, 3)."""

        altitude = float(np.float32(v.altitude_m))
        sun = _f32(v.sun_local)
        sky = self.sky_view(self.c.sky_view_lut_width, self.c.sky_view_lut_height, altitude, float(np.float32(_unit64(v.sun_local)[1])))
        disk, rays = _light(v).sun_disk_radiance, _rays(width, height, _f32(v.basis).cpu().numpy(), float(np.float32(v.tangent_half_fov)))
        flat = [a.reshape(width * height, -1) for a in (rays, scene, space, sid, position)]
        out = []
        for a in range(0, width * height, 1 << 20):
            d, color, space_, id_, pos = (x[a:a + (1 << 20)] for x in flat)
            color, space_, hit = color[:, :3].double(), space_[:, :3].double(), id_[:, 0] >= 0
            hdr = torch.empty_like(color)
            L, T = self.surface(altitude, d[hit], sun, pos[hit, :3].double().norm(dim=1))
            hdr[hit] = L + color[hit] * T
            hdr[~hit] = self.sky_pixel(sky, altitude, d[~hit], sun, color[~hit], space_[~hit], disk, v.tangent_half_fov, height)
            out.append(hdr.clamp_min(0.0))
        return torch.cat(out).reshape(width, height, 3)


def _unit64(v):
    v = np.asarray(v, np.float64)
    return v / np.linalg.norm(v)


def _shade64(images, v, sun_t, sky_l, ocean):
    """The surface shading of (W, H, 3) images: Lambert land, and the sea's
    specular, sky reflection and refracted seabed."""

    width, height = images["surface_id"].shape
    g = {n: t[..., :3].double() if t.dim() == 3 else t for n, t in images.items()}
    sun, e, (right, up, fwd) = _f32(v.sun_local), _f32(E), _f32(v.basis)
    sid = g["surface_id"]
    n = _unit(g["normal"])
    ndl = _dot(n, sun).clamp_min(0.0)[..., None]
    direct = e * sun_t * ndl
    land = g["albedo"] * (direct / math.pi + sky_l)
    background = torch.tensor([0.00015, 0.0002, 0.00035], dtype=torch.float64, device="cuda")
    color = torch.where((sid >= 0)[..., None], land, background)
    at = (sid == OCEAN_SURFACE_ID).nonzero(as_tuple=True)
    if not at[0].numel():
        return color
    pick = lambda name: g[name][at].double()  # noqa: E731
    n, ndl, direct, T, sky = n[at], ndl[at][:, 0], direct[at], sun_t[at], sky_l[at]
    pos = pick("position")
    view = -_unit(pos @ torch.stack([right, up, fwd]))
    ndv = _dot(n, view).clamp_min(1e-4)
    half = view + sun
    half = half / half.norm(dim=1, keepdim=True).clamp_min(1e-5)
    ndh, vdh = _dot(n, half).clamp_min(0.0), _dot(view, half).clamp_min(0.0)
    f0 = float(np.float32(ocean.dielectric_f0))
    fv, fs = f0 + (1.0 - f0) * (1.0 - ndv) ** 5, f0 + (1.0 - f0) * (1.0 - vdh) ** 5
    rough = float(np.float32(ocean.roughness))
    a2 = (rough ** 4 + pick("slope_variance") + math.tan(math.radians(SUN_DEG)) ** 2).clamp(1e-5, 1.0)
    den = ndh * ndh * (a2 - 1.0) + 1.0
    dist = a2 / (math.pi * den * den).clamp_min(1e-5)
    k = (a2.sqrt().sqrt() + 1.0) ** 2 / 8.0
    gv, gl = ndv / (ndv * (1.0 - k) + k).clamp_min(1e-5), ndl / (ndl * (1.0 - k) + k).clamp_min(1e-5)
    spec = e * T * (dist * gv * gl * fs * ndl / (4.0 * ndv * ndl).clamp_min(1e-4))[:, None]
    depth = pick("water_depth").clamp_max(ocean.max_visible_depth_m)
    bed_albedo, bed_normal = pick("seabed_albedo"), _unit(pick("seabed_normal"))
    inc, nv = _unit(pos), _unit(torch.stack([n @ right, n @ up, n @ fwd], 1))
    eta, ci = float(np.float32(1.0) / np.float32(ocean.refraction_index)), -_dot(inc, nv)
    cc = ci.clamp_min(0.0)
    disc = 1.0 - eta * eta * (1.0 - cc * cc)
    refr = torch.where((disc > 0.0)[:, None], _unit(inc * eta + nv * (eta * cc - disc.clamp_min(0.0).sqrt())[:, None]), inc)
    refr = _unit(inc * (1.0 - ocean.refraction_strength) + refr * ocean.refraction_strength)
    limit = 2.0 * ocean.max_visible_depth_m
    travel = (depth * ci.clamp_min(0.05) / (-_dot(refr, nv)).clamp_min(0.05)).clamp_max(limit)
    end = pos + refr * travel[:, None]
    live = (end[:, 2] > 0.1) & (ocean.refraction_strength > 0.0)
    z = end[:, 2].clamp_min(0.1)
    x, y = at[0].double(), at[1].double()
    sx = (end[:, 0] / (z * TF * width / height) * 0.5 + 0.5) * width - 0.5
    sy = (end[:, 1] / (z * TF) * 0.5 + 0.5) * height - 0.5
    dx, dy = sx - x, sy - y
    scale = (ocean.refraction_max_offset_pixels / (dx * dx + dy * dy).sqrt().clamp_min(1e-5)).clamp_max(1.0)
    sx, sy = x + dx * scale, y + dy * scale
    bx, by = sx.floor(), sy.floor()
    acc = {m: torch.zeros_like(pos) for m in ("albedo", "normal", "position")}
    weight = torch.zeros_like(sx)
    for oy in (0, 1):
        for ox in (0, 1):
            ix, iy = (bx + ox).long(), (by + oy).long()
            inside = (ix >= 0) & (ix < width) & (iy >= 0) & (iy < height)
            q = (ix.clamp(0, width - 1), iy.clamp(0, height - 1))
            p = g["terrain_position"][q]
            ok = inside & (g["terrain_surface_id"][q] >= 0) & (p[:, 2] > pos[:, 2] + 0.01) & ((p - pos).norm(dim=1) <= limit)
            w = torch.where(ok, (sx - bx if ox else 1.0 - (sx - bx)) * (sy - by if oy else 1.0 - (sy - by)), 0.0)
            for m in acc:
                acc[m] = acc[m] + g["terrain_" + m][q] * w[:, None]
            weight = weight + w
    found = live & (weight > 0.25)
    inv = (1.0 / weight.clamp_min(1e-9))[:, None]
    bed_albedo = torch.where(found[:, None], acc["albedo"] * inv, bed_albedo)
    bed_normal = torch.where(found[:, None], acc["normal"] / acc["normal"].norm(dim=1, keepdim=True).clamp_min(1e-30), bed_normal)
    depth = torch.where(found, (acc["position"] * inv - pos).norm(dim=1).clamp_max(ocean.max_visible_depth_m), depth)
    ext = _f32(ocean.absorption_per_m) + _f32(ocean.scattering_per_m)
    tr = (-ext * depth[:, None]).exp()
    bed = bed_albedo * (e * T * _dot(bed_normal, sun).clamp_min(0.0)[:, None] / math.pi + sky) * tr
    body = bed + (sky + direct / (4.0 * math.pi)) * (_f32(ocean.scattering_per_m) / ext) * (1.0 - tr)
    color[at] = body * (1.0 - fv)[:, None] + sky * fv[:, None] * ocean.sky_reflection_strength + spec
    return color


def _post64(case, hdr):
    """The display image of a (W, H, 3) float64 frame."""

    cfg = PostprocessConfig(bloom_passes=case["passes"])
    gain = 2.0 ** case["exposure_ev"] if case["tone_map"] else 1.0
    w, h = case["width"], case["height"]
    v = hdr * gain
    if case["bloom"] and case["passes"] > 0:
        hw, hh = max((w + 1) // 2, 1), max((h + 1) // 2, 1)
        xs, ys = torch.arange(hw, device="cuda") * 2, torch.arange(hh, device="cuda") * 2
        b = sum(v[(xs + i).clamp_max(w - 1)][:, (ys + j).clamp_max(h - 1)] for i in (0, 1) for j in (0, 1)) * 0.25
        bright = b.amax(2, keepdim=True)
        soft = (bright - cfg.bloom_threshold + cfg.bloom_knee).clamp(0.0, 2.0 * cfg.bloom_knee) ** 2 / max(4.0 * cfg.bloom_knee, 1e-6)
        b = b * torch.maximum(bright - cfg.bloom_threshold, soft) / bright.clamp_min(1e-6)
        b = b * (cfg.bloom_clamp / b.amax(2, keepdim=True).clamp_min(1e-6)).clamp_max(1.0)
        taps = [float(np.float32(t)) for t in (0.38774, 0.24477, 0.06136)]
        for _ in range(case["passes"]):
            for dim, size in ((0, hw), (1, hh)):
                at = torch.arange(size, device="cuda")
                b = sum(taps[abs(k)] * b.index_select(dim, (at + k).clamp(0, size - 1)) for k in (-2, -1, 0, 1, 2))
        px = (torch.arange(w, device="cuda").double() + 0.5) / w * hw - 0.5
        py = (torch.arange(h, device="cuda").double() + 0.5) / h * hh - 0.5
        x0, y0 = px.floor().long().clamp(0, hw - 1), py.floor().long().clamp(0, hh - 1)
        x1, y1 = (x0 + 1).clamp_max(hw - 1), (y0 + 1).clamp_max(hh - 1)
        fx, fy = (px - px.floor())[:, None, None], (py - py.floor())[None, :, None]
        low = b[x0][:, y0] * (1 - fx) + b[x1][:, y0] * fx
        high = b[x0][:, y1] * (1 - fx) + b[x1][:, y1] * fx
        v = v + (low * (1 - fy) + high * fy) * float(np.float32(cfg.bloom_strength))
    if not case["tone_map"]:
        return v.clamp(0.0, 1.0)
    v = v.clamp_min(0.0)
    m = (v * (2.51 * v + 0.03) / (v * (2.43 * v + 0.59) + 0.14)).clamp(0.0, 1.0)
    return torch.where(m <= 0.0031308, m * 12.92, 1.055 * m ** (1.0 / 2.4) - 0.055)


def _layers64(net):
    p = net.params().double()
    out, at = [], 0
    for o, i in layer_shapes(net.n_in, net.n_hidden, net.n_out):
        out.append([p[at:at + o * i].view(o, i).clone(), p[at + o * i:at + o * i + o].clone()])
        at += o * i + o
    return out


def _forward64(layers, x):
    for k, (w, b) in enumerate(layers):
        x = x @ w.T + b
        if k + 1 < len(layers):
            x = torch.nn.functional.silu(x)
    return x


def exact(case, seed):
    kind = case["kind"]
    with torch.no_grad():
        if kind in ("frame", "fused"):
            make, radius = PRESETS[case["preset"]]
            a, hdrs = Atmosphere64(make(), radius), []
            size = (case["width"], case["height"])
            for k, v in enumerate(_views(case, seed)):
                gb = _gbuffer(*size, v, seed, k)
                flat, hit = gb["position_view"].reshape(-1, 3), (gb["surface_id"] >= 0).reshape(-1)
                sun_t = torch.ones((flat.shape[0], 3), dtype=torch.float64, device="cuda")
                sky_l = torch.zeros_like(sun_t)
                sun_t[hit], sky_l[hit] = a.lighting(float(np.float32(v.altitude_m)), v.basis, _f32(v.sun_local), flat[hit])
                sun_t, sky_l = (t.reshape(*size, 3) for t in (sun_t, sky_l))
                if kind == "fused":
                    images = _shading_images(gb)
                    scene, sid = _shade64(images, v, sun_t, sky_l, OceanShading()).clamp_min(0.0), images["surface_id"]
                else:
                    scene, sid = gb["scene_hdr"], gb["surface_id"]
                hdrs.append(_as_layout(a.composite(v, scene, gb["space_hdr"], sid, gb["position_view"], *size), case))
            if kind == "fused":
                return hdrs
            out3 = dict(case, channels=3)  # the renderer's own lighting images have three channels
            return {"hdr": hdrs, "sun_t": _as_layout(sun_t, out3), "sky_l": _as_layout(sky_l, out3)}
        if kind == "sky" and case["mode"] != "net":
            make, radius = PRESETS[case["preset"]]
            a, v = Atmosphere64(make(), radius), _views(case, seed)[0]
            d = _rays(case["width"], case["height"], _f32(v.basis).cpu().numpy(), float(np.float32(TF))).reshape(-1, 3)
            sun, alt = _f32(v.sun_local), float(np.float32(v.altitude_m))
            if case["mode"] == "plain":
                L = a.sky_rays(torch.full_like(d[:, 0], alt), d, sun.expand_as(d))
            else:
                lut = a.sky_view(a.c.sky_view_lut_width, a.c.sky_view_lut_height, alt, float(np.float32(_unit64(v.sun_local)[1])))
                L = a.sky_tap(lut, alt, d, sun)
            return _as_layout(L.reshape(case["width"], case["height"], 3), case)
        if kind == "luts":
            make, radius = PRESETS[case["preset"]]
            a, v = Atmosphere64(make(), radius), frame_chain_cameras(seed)[0]
            c = a.c
            sky = a.sky_view(c.sky_view_lut_width, c.sky_view_lut_height, case["altitude_m"], float(np.float32(v.sun_local[1])))
            ap = a.slices(*a.columns(c.aerial_lut_width, c.aerial_lut_height, (16, 16), case["altitude_m"], v.sun_local,
                                     v.basis, TF), c.aerial_lut_depth)
            ap = ap.reshape(c.aerial_lut_depth, c.aerial_lut_height, c.aerial_lut_width, 3)
            return [t.transpose(0, 1).contiguous() for t in (a.t, a.m, sky)] + [ap.permute(2, 1, 0, 3).contiguous()]
        if kind == "batch":
            jobs = _batch_jobs(case, seed)
            offsets, total = BatchedLutBuilder.layout(jobs)
            arena = torch.zeros((total, 4), dtype=torch.float64, device="cuda")
            for k, (config, radius) in enumerate(batched_lut_sets()):
                a = Atmosphere64(config, radius)
                mine = [(j, o) for j, o in zip(jobs, offsets) if j.param_set == k]
                for depth in sorted({j.depth for j, _ in mine}):  # sky-view jobs: depth 1; aerial sides from 16
                    same = [(j, o) for j, o in mine if j.depth == depth]
                    if depth == 1:
                        rays = [a.sky_texels(j.width, j.height, j.camera_altitude_m, j.sun_zenith_cosine) for j, _ in same]
                        L = a.sky_rays(*(torch.cat(t) for t in zip(*rays)))[None]
                    else:
                        rays = [a.columns(j.width, j.height, (j.frame_width, j.frame_height), j.camera_altitude_m,
                                          j.sun_local, j.view_basis, j.tangent_half_fov) for j, _ in same]
                        L = a.slices(*(torch.cat(t) for t in zip(*rays)), depth)
                    at = 0
                    for j, o in same:
                        n = j.width * j.height
                        arena[o:o + n * depth, :3] = L[:, at:at + n].reshape(-1, 3)
                        at += n
            return arena
        if kind == "post":
            return _as_layout(_post64(case, _hdr_image(case, seed).double()), case)
        if kind == "evaluate":
            net = _network(_shape(case), seed)
            y = _forward64(_layers64(net), _train_set(_shape(case), case["samples"], seed, False)[0].double())
            return {"f32": y, "bf16": y}
    if kind == "train":
        net = Mlp(*_shape(case), seed=seed % (1 << 31))
        layers = _layers64(net)
        leaves = [t.requires_grad_() for pair in layers for t in pair]
        x, y, w = _train_set(_shape(case), case["samples"], seed, case["weighted"])
        err = (_forward64(layers, x.double()) - y.double()) ** 2
        loss = (err if w is None else err * w.double()).sum()
        grads = torch.autograd.grad(loss / err.numel(), leaves)
        # the first Adam step: both bias-corrected moments are the gradient's own
        lr, eps = float(np.float32(1e-3)), float(np.float32(1e-8))
        return {"loss": loss.detach().reshape(1),
                "params": torch.cat([(p.detach() - lr * g / (g.abs() + eps)).reshape(-1) for p, g in zip(leaves, grads)])}
    # No 64-bit value: the surrogate composite and the sky network answer with 16-bit networks and a seeded check of
    # their own; a raster's and a whole frame's pixels follow from coverage rules in snapped float32 coordinates.
    return None
