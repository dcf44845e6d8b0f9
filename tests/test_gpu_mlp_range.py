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


@pytest.mark.parametrize("n_in", [11, 16])
def test_infinite_output_biases_of_the_tensor_core_forward(n_in):
    """The bias rides in three parts: an infinite one is its first part alone."""

    import torch

    from planet_renderer_gb300.atmosphere.mlp import Mlp

    net = Mlp(n_in, 2, 3, seed=3)
    p = net.params()
    p[-3:] = torch.tensor([float("inf"), 0.5, float("-inf")], device="cuda")
    net.set_params(p)
    x = torch.as_tensor(np.random.default_rng(2).uniform(-1.0, 1.0, (130, n_in)).astype(np.float32), device="cuda")
    got = net.forward(x, "bf16_tc")
    assert torch.isposinf(got[:, 0]).all() and torch.isfinite(got[:, 1]).all() and torch.isneginf(got[:, 2]).all()
    net.close()
