"""Training samples' features against the numbers they are drawn from: a
sample draws its features, forms the geometry in float32 and returns the
features of that geometry."""

from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

F = np.float32


def _drawn(seed, n, k):
    """The sample generator's counter-based uniforms, as features in -1..1."""

    with np.errstate(over="ignore"):
        z = np.uint64(seed) + np.uint64(0x9E3779B97F4A7C15) * (np.arange(n, dtype=np.uint64) * np.uint64(16) + np.uint64(k + 1))
        z = (z ^ (z >> np.uint64(30))) * np.uint64(0xBF58476D1CE4E5B9)
        z = (z ^ (z >> np.uint64(27))) * np.uint64(0x94D049BB133111EB)
        z ^= z >> np.uint64(31)
    return F(2.0) * ((z >> np.uint64(40)).astype(F) * F(2.0 ** -24)) - F(1.0)


@pytest.mark.parametrize("kind", [0, 1])
def test_altitude_and_view_features(kind):
    from planet_renderer_gb300.atmosphere.surrogate import SampleSource, parameter_grid

    n, seed = 1 << 18, 5
    src = SampleSource(parameter_grid()[:1])
    x = src.samples(kind, n, seed)[0].cpu().numpy()
    top = F(src.top_altitude_m)
    src.close()
    # the altitude feature is 2 sqrt(h / top) - 1 in IEEE operations
    d0 = _drawn(seed, n, 1)
    h = top * F(0.25) * (d0 + F(1.0)) * (d0 + F(1.0))
    np.testing.assert_array_equal(x[:, 0], F(2.0) * np.sqrt(np.clip(h * F(1.0 / float(top)), F(0.0), F(1.0))) - F(1.0))
    # the view feature is the root of a difference of two angles, each rounded to 2^-24 of its size (between 1 and
    # pi: 2/3 of 2^-24 in the mean for the two); the root makes that 1/2 / (pi/2 x) of it, 8/pi in the mean over x
    # down to 3e-4, where the difference is its own rounding: 1.0e-7, 1.3e-7 with the feature's, and half as much
    # again for an arc cosine that is not correctly rounded
    assert np.abs(x[:, 1].astype(np.float64) - _drawn(seed, n, 2)).mean() <= 2.0e-7
