"""The splits of a march over lanes, chosen by size, at the sizes where each
begins and ends: frames and LUTs of every lane count against the oracle."""

from __future__ import annotations

import dataclasses

import numpy as np
import pytest

from conftest import CUTOFF_MARGIN_M, assert_exact_parity, assert_parity, exact_parity_violations

pytestmark = pytest.mark.gpu

R = 6_360_000.0
E = (4.0, 3.9, 3.7)


def _frame(width, height, layout):
    import torch

    from oracle.atm import OracleAtmosphere, sun_disk_radiance
    from planet_renderer_gb300 import camera
    from planet_renderer_gb300.atmosphere import AtmosphereRenderer, scene
    from planet_renderer_gb300.atmosphere.config import earth_baseline

    basis, tanfov = camera.view_basis(0.0, -20.0), camera.tangent_half_fov(60.0)
    sun = camera.sun_from_zenith(80.0, 40.0)
    cfg, cr = earth_baseline(), R + 20_000.0
    gb = scene.synthesize_gbuffer(width, height, R, 20_000.0, basis, tanfov, sun, seed=5, device="cuda")
    disk = sun_disk_radiance(E, 0.266)
    lay = (lambda t: t) if layout == "wh" else (lambda t: t.transpose(0, 1).contiguous())
    r = AtmosphereRenderer(width, height, cfg, layout=layout)
    r.update(R, cr, sun.copy(), E, 0.266)
    hdr = torch.zeros_like(lay(gb["scene_hdr"]))
    args = (R, cr, sun, E, disk, 0.266, basis, tanfov, 4.0, 12.0)
    images = [lay(gb[k]) for k in ("scene_hdr", "space_hdr", "surface_id", "position_view")]
    r.composite(*images, hdr, *args)
    host = {k: v.cpu().numpy() for k, v in gb.items()}
    margin = np.full((width, height), np.inf)

    def oracle(precision):
        o = OracleAtmosphere(width, height, cfg, precision)
        o.update(R, cr, sun.copy(), E, 0.266)
        return o.composite(host["scene_hdr"], host["space_hdr"], host["surface_id"], host["position_view"], *args,
                           margin_out=margin)[0]

    return r, images, args, hdr, oracle, margin


# 16, 8, 4, 2 lanes a pixel and 1, at a first and a last size, odd ones; one pixel
@pytest.mark.parametrize("width,height", [(1, 1), (96, 76), (97, 76), (151, 97), (171, 171), (243, 241), (343, 341)])
@pytest.mark.parametrize("layout", ["wh", "hw"])
def test_frame_matches_oracle_at_each_lane_count(width, height, layout):
    _, _, _, hdr, oracle, margin = _frame(width, height, layout)
    got = hdr.cpu().numpy() if layout == "wh" else hdr.transpose(0, 1).cpu().numpy()
    f32, f64 = oracle("f32"), oracle("f64")
    # the frames' criterion: exact parity, but for rare pixels with a sample at a density cutoff
    bad = exact_parity_violations(got, f32, f64).any(axis=-1)
    assert (margin[bad] < CUTOFF_MARGIN_M).all() and bad.mean() <= 1e-4
    assert_exact_parity(got[~bad], f32[~bad], f64[~bad], f"{width}x{height} {layout}")


# network tiles of 128 pixels, 16 along the contiguous axis by 8: whole, partial, a single pixel
@pytest.mark.parametrize("width,height", [(1, 1), (16, 8), (17, 9), (130, 97)])
@pytest.mark.parametrize("layout", ["wh", "hw"])
def test_checked_surrogate_equals_plain_at_tile_edges(width, height, layout):
    """Every network pixel re-integrated: the frame is the plain composite's."""

    import torch

    from planet_renderer_gb300.atmosphere.mlp import Mlp
    from planet_renderer_gb300.atmosphere.surrogate import Surrogate

    r, images, args, hdr, _, _ = _frame(width, height, layout)
    got = torch.zeros_like(hdr)
    r.composite_surrogate(*images, got, *args, surrogate=Surrogate(Mlp(11, 4, 6, seed=5), None), check_fraction=1.0)
    np.testing.assert_allclose(got.cpu().numpy(), hdr.cpu().numpy(), rtol=2e-5, atol=1e-9)


# sky-view texels by 8, 4, 2 lanes and 1; multi-scattering directions by 4 lanes and 1
@pytest.mark.parametrize("sky,ms,dirs", [((16, 17), (8, 8), 4), ((192, 108), (32, 32), 64), ((257, 150), (33, 31), 65),
                                         ((300, 301), (48, 47), 128)])
def test_luts_match_oracle_at_each_lane_count(sky, ms, dirs, oracle_f32):
    from planet_renderer_gb300.atmosphere import AtmosphereRenderer
    from planet_renderer_gb300.atmosphere.config import earth_baseline

    cfg = dataclasses.replace(earth_baseline(), sky_view_lut_width=sky[0], sky_view_lut_height=sky[1],
                              multi_scattering_lut_width=ms[0], multi_scattering_lut_height=ms[1],
                              multi_scattering_directions=dirs, sky_view_steps=27, aerial_lut_depth=70)
    r = AtmosphereRenderer(16, 9, cfg)
    kw = dict(planet_radius_m=R, camera_altitude_m=500.0, sun_zenith_cosine=0.25, sun_local=(0.9682458, 0.25, 0.0))
    for kind in ("transmittance", "multi_scattering", "sky_view", "aerial"):
        r.build_lut(kind, **kw)
    ar = float(np.float32(np.radians(0.266)))
    t = oracle_f32.build_transmittance(cfg, R)
    m = oracle_f32.build_multi_scattering(cfg, R, E, ar, t)
    assert_parity(r.multi_scattering_lut.to_numpy(), m, "multi-scattering")
    assert_parity(r.sky_view_lut.to_numpy(), oracle_f32.build_sky_view(cfg, R, 500.0, 0.25, E, ar, t, m), "sky-view")
    basis = ((1.0, 0.0, 0.0), (0.0, 1.0, 0.0), (0.0, 0.0, 1.0))
    ap = oracle_f32.build_aerial(cfg, 16, 9, R, 500.0, (0.9682458, 0.25, 0.0), E, ar, basis, np.tan(np.pi / 6), t, m)
    assert_parity(r.aerial_scattering_lut.to_numpy(), ap, "aerial, three slices a lane")


# segments of optical thickness below 1/4, across it, across 1 and beyond: steps of a few to 80 km
@pytest.mark.parametrize("scale", [0.0, 1.0, 6.0, 40.0, 2000.0])
def test_segments_of_every_thickness(scale, oracle_f32):
    from planet_renderer_gb300.atmosphere import AtmosphereRenderer
    from planet_renderer_gb300.atmosphere.config import earth_baseline

    cfg = earth_baseline()
    cfg = dataclasses.replace(cfg, sky_view_lut_width=32, sky_view_lut_height=24, sky_view_steps=12,
                              rayleigh_scattering_per_m=tuple(scale * v for v in cfg.rayleigh_scattering_per_m))
    r = AtmosphereRenderer(16, 9, cfg)
    kw = dict(planet_radius_m=R, camera_altitude_m=500.0, sun_zenith_cosine=0.25, sun_local=(0.9682458, 0.25, 0.0))
    for kind in ("transmittance", "multi_scattering", "sky_view"):
        r.build_lut(kind, **kw)
    ar = float(np.float32(np.radians(0.266)))
    t = oracle_f32.build_transmittance(cfg, R)
    m = oracle_f32.build_multi_scattering(cfg, R, E, ar, t)
    assert_parity(r.multi_scattering_lut.to_numpy(), m, "multi-scattering")
    assert_parity(r.sky_view_lut.to_numpy(), oracle_f32.build_sky_view(cfg, R, 500.0, 0.25, E, ar, t, m), "sky-view")


@pytest.mark.parametrize("n_in", [12, 13, 14])
def test_tcgen05_bias_inputs(n_in):
    """The bias's three inputs beside the network's (13 leave room) and in a step of their own (14 do not)."""

    import torch

    from oracle import mlp_fp64
    from planet_renderer_gb300.atmosphere.mlp import Mlp, layer_shapes

    net = Mlp(n_in, 2, 3, seed=3)
    p = net.params()
    p += torch.linspace(-0.3, 0.3, p.numel(), device="cuda")  # biases are zero at first
    net.set_params(p)
    x = np.random.default_rng(2).uniform(-1.0, 1.0, (130, n_in)).astype(np.float32)
    got = net.forward(torch.as_tensor(x, device="cuda"), "bf16_tc").cpu().numpy()
    ref = mlp_fp64.forward(p.cpu().numpy(), layer_shapes(n_in, 2, 3), x)
    scale = np.sqrt(np.mean(ref ** 2))
    assert np.sqrt(np.mean((got - ref) ** 2)) <= 2e-2 * scale  # bf16 operands, as the forward's own test
    net.close()
