"""The polynomials of a segment's in-scattering weight, on the kernels' own
coefficients (no GPU)."""

from __future__ import annotations

import re
from pathlib import Path

import numpy as np
import pytest

SOURCE = Path(__file__).resolve().parents[1] / "planet-real-time-render_gb300" / "csrc" / "atm_device.cuh"


@pytest.mark.parametrize("name,end", [("phi_quarter", 0.25), ("phi_one", 1.0)])
def test_polynomial_is_within_its_bound(name, end):
    """phi(x) = (1 - e^-x) / x, in 64 bits: within 3e-9 with the float coefficients, 1 at 0."""

    body = re.search(name + r"\(float x\) \{(.*?)\n\}", SOURCE.read_text(), re.S).group(1)
    c = [float(np.float32(v)) for v in re.findall(r"(-?\d+\.\d+)f", body)]
    c.sort(key=abs)  # 1, -1/2, 1/6, ...: falling in size with the power
    assert c[-1] == 1.0
    x = np.linspace(0.0, end, 200_001)[1:]
    assert np.abs(np.polyval(c, x) / (-np.expm1(-x) / x) - 1.0).max() <= 3e-9
