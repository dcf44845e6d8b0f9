"""Kernels whose blocks are runs of 32 pixels by 8 rows, at the edges of a
run and of a block, in both layouts, against the oracles."""

from __future__ import annotations

import numpy as np
import pytest

from test_gpu_ocean import _check, _frame, _run

pytestmark = pytest.mark.gpu

SIZES = [(1, 1), (32, 8), (33, 9), (7, 65)]


@pytest.mark.parametrize("width,height", SIZES)
@pytest.mark.parametrize("resolution,layout", [(32, "wh"), (64, "hw"), (128, "wh"), (256, "hw")])
def test_ocean_at_run_edges_and_each_spectrum_size(width, height, resolution, layout):
    from oracle import ocean
    from planet_renderer_gb300 import camera as cam

    config = {"spectrum_resolution": resolution, "geometry_cascades": 3}
    inputs = _frame(width, height, 5)
    q = np.linalg.qr(np.random.default_rng(3).normal(size=(3, 3)))[0]
    a = {"planet_radius_m": 6_371_000.0, "camera_altitude_m": 9.0,
         "planet_frame": (q[:, 0], q[:, 1], np.cross(q[:, 0], q[:, 1])), "view_basis": cam.view_basis(30.0, -40.0),
         "tangent_half_fov": cam.tangent_half_fov(60.0), "time_seconds": 3.5, "debug_mode": 0}
    ref, _ = ocean.rasterize(inputs, ocean.OceanSettings(**config), a["planet_radius_m"], 9.0, a["planet_frame"],
                             a["view_basis"], a["tangent_half_fov"], a["time_seconds"], 0)
    got, _ = _run(inputs, config, a, layout, 3)
    _check(got, ref)


# blur strips of 24 (two passes) and 28 (one) half-resolution texels, segments of rows, one texel; odd passes
@pytest.mark.parametrize("width,height", [(1, 1), (2, 5), (48, 9), (49, 131), (57, 113), (400, 3)])
@pytest.mark.parametrize("layout", ["wh", "hw"])
@pytest.mark.parametrize("passes", [1, 2, 3, 8])
def test_bloom_at_strip_and_segment_edges(width, height, layout, passes):
    from types import SimpleNamespace

    from oracle import postprocess as op
    from test_gpu_postprocess import DEFAULTS, DISPLAY_ATOL, _processor
    from test_gpu_postprocess import _run as _process

    hdr = np.exp(np.random.default_rng(width).normal(0.0, 1.5, (width, height, 3))).astype(np.float32)
    config = dict(bloom_passes=passes)
    cfg = SimpleNamespace(**{**DEFAULTS, **config})
    pp = _processor(width, height, config, layout)
    got = _process(pp, hdr, 1.0, True, True, layout=layout)
    a = op.extract(hdr, float(np.float32(2.0)), cfg)
    for _ in range(passes):
        a = op.blur_vertical(op.blur_horizontal(a))
    np.testing.assert_allclose(pp.bloom_plane().cpu().numpy(), a, rtol=2.0 ** -22, atol=0)
    np.testing.assert_allclose(got, op.process(hdr, 1.0, cfg, bloom=True, tone_map=True), rtol=0, atol=DISPLAY_ATOL)
    pp.close()


def test_display_of_the_largest_values():
    """The ACES fit's quotient where its terms near and leave float's range: the IEEE quotient's result."""

    from types import SimpleNamespace

    from oracle import postprocess as op
    from test_gpu_postprocess import DEFAULTS, DISPLAY_ATOL, _processor

    v = np.array([0.0, 1e-30, 1e-3, 0.0031, 1.0, 9e17, 1.1e18, 1.15e19, 1.18e19, 1.3e19, 3e38, np.inf, np.nan, -1.0],
                 np.float32)
    hdr = np.repeat(v[:, None, None], 3, 2)
    cfg = SimpleNamespace(**DEFAULTS)
    pp = _processor(len(v), 1, {})
    with np.errstate(all="ignore"):
        ref = op.process(hdr, 0.0, cfg, bloom=False, tone_map=True)
    ref = np.where(np.isnan(ref), np.float32(0.0), ref)  # the device's clamps take the bound for a NaN
    np.testing.assert_allclose(_process_nan(pp, hdr), ref, rtol=0, atol=DISPLAY_ATOL)
    pp.close()


def _process_nan(pp, hdr):
    import torch

    src = torch.as_tensor(hdr, device="cuda")
    display = torch.full_like(src, -1.0)
    pp.process(src, display, 0.0, bloom=False, tone_map=True)
    return display.cpu().numpy()


# an odd number of depth keys; boxes of a few pixels, of a warp, of several tiles; fewer triangles than a warp's
@pytest.mark.parametrize("width,height,patches,res", [(1, 1, 3, 1), (31, 33, 4, 12), (263, 41, 3, 2), (701, 397, 2, 1)])
@pytest.mark.parametrize("layout", ["wh", "hw"])
def test_raster_boxes_of_each_size(width, height, patches, res, layout):
    from oracle import raster
    from test_gpu_raster import _compare, _mesh_tensors, _render, _terrain

    view, normal, material, height_m, cell, tris, skirt, level, surface = _terrain(patches, res, 3)
    active = list(range(patches))
    ref = raster.render(view, normal, material, height_m, cell, tris, active, 0.5, 0.62, width, height, 0, level,
                        surface, res, skirt)
    ref["material_weights"] = ref.pop("material")
    mesh = _mesh_tensors(view, normal, material, height_m, cell, tris, active, skirt, level, surface, res)
    got, count = _render(mesh, width, height, 0.5, 0.62, 0, layout)
    assert count == ref["clipped_count"]
    _compare(got, ref, ref["ties"])
