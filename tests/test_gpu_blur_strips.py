"""The streaming bloom blur (planes above 196,608 half-resolution texels) at
the edges of its strips (56 texels of two passes, 60 of one; four a block) and
of its segments, in both layouts, against the oracle.  Smaller planes are
blurred by tiles of 32 x 8 texels, which the other post-process tests cover."""

from __future__ import annotations

from types import SimpleNamespace

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SMALL_PLANE = 3 << 16


def _compare(width, height, layout, passes):
    from oracle import postprocess as op
    from test_gpu_postprocess import DEFAULTS, DISPLAY_ATOL, _processor, _run

    hdr = np.exp(np.random.default_rng(width).normal(0.0, 1.5, (width, height, 3)).astype(np.float32))
    config = dict(bloom_passes=passes)
    cfg = SimpleNamespace(**{**DEFAULTS, **config})
    pp = _processor(width, height, config, layout)
    got = _run(pp, hdr, 1.0, True, True, layout=layout)
    a = op.extract(hdr, float(np.float32(2.0)), cfg)
    for _ in range(passes):
        a = op.blur_vertical(op.blur_horizontal(a))
    np.testing.assert_allclose(pp.bloom_plane().cpu().numpy(), a, rtol=2.0 ** -22, atol=0)
    np.testing.assert_allclose(got, op.process(hdr, 1.0, cfg, bloom=True, tone_map=True), rtol=0, atol=DISPLAY_ATOL)
    pp.close()


@pytest.mark.parametrize("fast", [1, 2, 3, 56, 57, 60, 61, 224, 225, 240, 241, 673])
@pytest.mark.parametrize("layout", ["wh", "hw"])
@pytest.mark.parametrize("passes", [1, 2])
def test_strip_edges(fast, layout, passes):
    slow = SMALL_PLANE // fast + 1  # the first plane past the tiles
    frame = (2 * fast - 1, 2 * slow) if layout == "hw" else (2 * slow, 2 * fast - 1)
    _compare(*frame, layout, passes)


# the last plane of the tiles; segments of the shortest and of longer lengths, several blocks of strips, odd passes
@pytest.mark.parametrize("width,height,passes", [(1024, 768, 3), (1026, 768, 3), (3840, 2160, 4), (2561, 1439, 1)])
@pytest.mark.parametrize("layout", ["wh", "hw"])
def test_large_planes(width, height, layout, passes):
    _compare(width, height, layout, passes)
