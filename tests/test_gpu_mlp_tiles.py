"""FP32 network tiles of 64 samples at their edges: gradients, an optimiser
step and the forward of ragged batches, one tile to several a block, for every
hidden-layer count and the smallest and largest inputs and outputs."""

from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(1, 1, 1), (16, 2, 8), (5, 3, 7), (13, 4, 2)])
@pytest.mark.parametrize("n", [1, 63, 64, 65, 12_000])
def test_gradient_step_and_forward_at_tile_edges(shape, n):
    import torch

    from oracle import mlp_fp64
    from planet_renderer_gb300.atmosphere.mlp import Mlp, layer_shapes

    net = Mlp(*shape, seed=4)
    rng = np.random.default_rng(n)
    x = rng.uniform(-1.0, 1.0, (n, shape[0])).astype(np.float32)
    t = rng.normal(0.0, 1.0, (n, shape[2])).astype(np.float32)
    w = rng.uniform(0.1, 2.0, (n, shape[2])).astype(np.float32)
    xd, td, wd = (torch.as_tensor(a, device="cuda") for a in (x, t, w))
    p = net.params().cpu().numpy().astype(np.float64)
    shapes = layer_shapes(*shape)
    y = mlp_fp64.forward(p, shapes, x)
    assert np.max(np.abs(net.forward(xd).cpu().numpy() - y)) <= 1e-5 * np.abs(y).max()
    ref = mlp_fp64.gradient(p, shapes, x, t, w)
    g, sq = net.gradient(xd, td, wd)
    assert np.max(np.abs(g.cpu().numpy() - ref)) <= 1e-4 * np.abs(ref).max()
    assert abs(float(sq) - np.sum(w * (y - t) ** 2)) <= 1e-4 * float(sq)
    # the first Adam step moves each parameter by lr g / (|g| + eps): the step's gradient is gradient()'s
    gd = g.cpu().numpy().astype(np.float64)
    loss = net.train_step(xd, td, lr=1e-3, weights=wd)
    assert float(loss) == float(sq)
    np.testing.assert_allclose(net.params().cpu().numpy(), p - 1e-3 * gd / (np.abs(gd) + 1e-8), rtol=0, atol=2e-7)
    net.close()
