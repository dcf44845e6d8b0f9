"""Shells of uniform density: scale heights so large that the exponent of the
density is 0 all the way up."""

from __future__ import annotations

import dataclasses

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _luts(height_m, radius, altitude_m):
    from planet_renderer_gb300.atmosphere import AtmosphereRenderer
    from planet_renderer_gb300.atmosphere.config import earth_baseline

    cfg = dataclasses.replace(earth_baseline(), rayleigh_scale_height_m=height_m, mie_scale_height_m=height_m)
    r = AtmosphereRenderer(16, 9, cfg)
    kw = dict(planet_radius_m=radius, camera_altitude_m=altitude_m, sun_zenith_cosine=0.05, sun_local=(0.99875, 0.05, 0.0))
    out = []
    for kind, field in (("transmittance", r.transmittance_lut), ("multi_scattering", r.multi_scattering_lut),
                        ("sky_view", r.sky_view_lut), ("aerial", r.aerial_scattering_lut)):
        r.build_lut(kind, **kw)
        out.append(field.to_numpy())
    r.close()
    return out


@pytest.mark.parametrize("radius", [50_000.0, 6_360_000.0])
@pytest.mark.parametrize("altitude_m", [0.0, 3.0, 2000.0, 2.0e6])
def test_larger_scale_heights_change_nothing(radius, altitude_m):
    """At 1e30 m the density is 1 to the last bit throughout; 1e60 m is the same shell."""

    for a, b in zip(_luts(1e30, radius, altitude_m), _luts(1e60, radius, altitude_m)):
        assert np.isfinite(b).all()
        np.testing.assert_array_equal(a, b)
