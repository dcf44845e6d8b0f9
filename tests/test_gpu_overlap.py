"""Fused frames whose output is also an input: every pixel is read before it
is written, with and without the networks."""

from __future__ import annotations

import numpy as np
import pytest

from test_gpu_frame import _frame, _separate

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shared", ["space_hdr", "position", "albedo", "terrain_normal"])
@pytest.mark.parametrize("layout", ["wh", "hw"])
@pytest.mark.parametrize("nets", [False, True])
def test_hdr_may_be_an_input_of_the_fused_frame(shared, layout, nets):
    import torch

    from planet_renderer_gb300.atmosphere.mlp import Mlp
    from planet_renderer_gb300.atmosphere.surrogate import Surrogate

    # the stars show from space
    r, images, args, v = _frame(131, 70, 2_000_000.0 if shared == "space_hdr" else 2000.0, 40.0, 30.0, layout)
    sg = Surrogate(Mlp(11, 4, 6, seed=5), Mlp(10, 3, 3, seed=6)) if nets else None
    ref = _separate(r, images, args, v, surrogate=sg)
    own = {k: t.clone() for k, t in images.items()}
    hdr = own[shared]
    space = own.pop("space_hdr")
    r.render_frame(own, space, hdr, *args, surrogate=sg, check_fraction=0.0, seed=3)
    torch.cuda.synchronize()
    # the tolerance of the fused frame's own test
    np.testing.assert_allclose(hdr.cpu().numpy(), ref, rtol=1e-5, atol=1e-9)
    r.close()
