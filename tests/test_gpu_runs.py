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
