"""Batched aerial volumes on either side of the rule by which lanes share a
column: few columns (8 or 32 lanes by depth, odd depths, partial groups) and
many (a lane each), against the single-LUT kernel."""

from __future__ import annotations

import dataclasses

import numpy as np
import pytest

from conftest import assert_parity

pytestmark = pytest.mark.gpu

SIZES = [(4, 4, 8), (5, 7, 9), (16, 16, 31), (33, 9, 32), (9, 5, 33), (31, 5, 65), (7, 11, 256)]


@pytest.mark.parametrize("fill", [0, 40])
@pytest.mark.parametrize("tuning", [(16, 4, 3), (1, 1, 1), (33, 4096, 8)])
def test_columns_shared_by_lanes(fill, tuning):
    """`fill` volumes of 64 x 64 columns put the batch past the rule's line."""

    import torch

    from planet_renderer_gb300.atmosphere import AtmosphereRenderer
    from planet_renderer_gb300.atmosphere.batch import AERIAL, SKY_VIEW, BatchedLutBuilder, BatchJob, Tuning
    from planet_renderer_gb300.atmosphere.workloads import batched_lut_sets

    sets = batched_lut_sets()
    kw = dict(camera_altitude_m=900.0, sun_local=(0.6, 0.8, 0.0))
    jobs = [BatchJob(AERIAL, k & 1, w, h, d, **kw) for k, (w, h, d) in enumerate(SIZES)]
    jobs.append(BatchJob(SKY_VIEW, 0, 17, 16, camera_altitude_m=900.0, sun_zenith_cosine=0.8))
    jobs += [BatchJob(AERIAL, 0, 64, 64, 8, **kw)] * fill
    builder = BatchedLutBuilder(sets)
    builder.samples(reset=True)
    result = builder.build(jobs, Tuning(*tuning), arena=torch.full((sum(j.texels for j in jobs), 4), -1.0, device="cuda"))
    torch.cuda.synchronize()
    samples = builder.samples(reset=True)
    expected = {}
    for i, j in enumerate(jobs):
        cfg, radius = sets[j.param_set]
        if i < len(SIZES) or j.kind == SKY_VIEW or j.depth not in expected:
            cfg = dataclasses.replace(cfg, aerial_lut_width=j.width, aerial_lut_height=j.height,
                                      aerial_lut_depth=max(j.depth, 8))
            if j.kind == SKY_VIEW:
                cfg = dataclasses.replace(cfg, sky_view_lut_width=j.width, sky_view_lut_height=j.height)
            r = AtmosphereRenderer(j.frame_width, j.frame_height, cfg)
            r.build_lut("transmittance", planet_radius_m=radius)
            r.build_lut("multi_scattering", planet_radius_m=radius)
            r.radiance_samples(reset=True)
            r.build_lut("sky_view" if j.kind == SKY_VIEW else "aerial", planet_radius_m=radius, **kw,
                        sun_zenith_cosine=0.8, view_basis=j.view_basis, tangent_half_fov=j.tangent_half_fov)
            field = r.sky_view_lut if j.kind == SKY_VIEW else r.aerial_scattering_lut
            expected[i if i <= len(SIZES) else j.depth] = field.to_numpy(), r.radiance_samples(reset=True)
            r.close()
        ref, n = expected[i if i <= len(SIZES) else j.depth]
        samples -= n
        # the tolerance of the batch's own test: the same device functions, composed in another order
        assert_parity(result.lut(i).cpu().numpy(), ref, f"job {i} {j.width}x{j.height}x{j.depth}", rtol=1e-4,
                      atol_frac=1e-6)
    assert samples == 0
    builder.close()
