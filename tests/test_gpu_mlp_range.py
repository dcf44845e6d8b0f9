"""Network forwards at the ends of float's range."""

from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("z", [-3e38, -1e32, -1e4, -104.0, -88.5, -87.0, -80.5, -20.0, 0.0, 20.0, 1e32])
def test_silu_of_large_preactivations(z):
    """One hidden neuron at z: below -87.3 the SiLU's size is under 1e-36."""

    import torch

    from planet_renderer_gb300.atmosphere.mlp import HIDDEN, Mlp

    net = Mlp(1, 1, 1, seed=0)
    p = torch.zeros_like(net.params())
    p[0], p[2 * HIDDEN] = z, 1.0  # W1[0][0] and W2[0][0]
    net.set_params(p)
    x = torch.ones((70, 1), device="cuda")
    z = float(np.float32(z))
    with np.errstate(over="ignore"):
        ref = z / (1.0 + np.exp(np.float64(-z)))
    np.testing.assert_allclose(net.forward(x, "f32").cpu().numpy(), ref, rtol=1e-6, atol=2e-36)
    net.close()
