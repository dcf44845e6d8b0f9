"""The display transform's error against 64 bits."""

from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

F = np.float32


def test_no_further_from_float64_than_a_correctly_rounded_power():
    """The ACES fit and sRGB segment over their range: no larger an error, rms,
    than the reference's float32 operations with a correctly rounded power."""

    import torch

    from test_gpu_postprocess import _processor

    v = np.geomspace(1e-3, 40.0, 300_000).astype(F)
    pp = _processor(1000, 100, {})
    hdr = torch.as_tensor(v.reshape(1000, 100, 3), device="cuda")
    display = torch.empty_like(hdr)
    pp.process(hdr, display, 0.0, bloom=False, tone_map=True)
    got = display.cpu().numpy().reshape(-1).astype(np.float64)
    pp.close()
    a, b, c, d, e = 2.51, 0.03, 2.43, 0.59, 0.14

    def fit(x, cast):
        a_, b_, c_, d_, e_ = (cast(k) for k in (a, b, c, d, e))
        return np.clip(x * (a_ * x + b_) / (x * (c_ * x + d_) + e_), 0, 1)

    m32 = fit(v, F)
    rounded = F(1.055) * np.power(m32.astype(np.float64), float(F(1.0 / 2.4))).astype(F) - F(0.055)
    exact = 1.055 * np.power(fit(v.astype(np.float64), np.float64), 1.0 / 2.4) - 0.055
    segment = (m32 > F(0.0031308)) & (m32 < 1)

    def rms(x):
        return float(np.sqrt(np.mean(((x - exact) / exact)[segment] ** 2)))

    assert rms(got) <= rms(rounded.astype(np.float64)), (rms(got), rms(rounded.astype(np.float64)))
