"""The raster of a stream so large that its listed triangles and their tiles do
not fit one 64-bit counter: the tile counts' prefix comes from the scans then.
The frame must be the one that a small stream gives."""

from __future__ import annotations

import pytest

pytestmark = pytest.mark.gpu

WIDTH, HEIGHT = 16384, 4096
TILES = ((WIDTH - 1) // 256 + 2) * ((HEIGHT - 1) // 32 + 2)  # a triangle's, at most


@pytest.mark.parametrize("resolution,altitude_m", [(1, 40.0), (6, 900.0)])
def test_frame_of_a_stream_past_the_counter(resolution, altitude_m):
    import torch

    from planet_renderer_gb300 import camera
    from planet_renderer_gb300.raster import TerrainRaster, synthetic_terrain

    if torch.cuda.mem_get_info()[0] < 40 << 30:
        pytest.skip("the stream takes 9 GB, the two G-buffers 10 GB")
    tf = camera.tangent_half_fov(60.0)
    mesh = synthetic_terrain(WIDTH, HEIGHT, tf, altitude_m=altitude_m, rows=5, columns=7, resolution=resolution,
                             relief_m=50.0, base_height_m=0.0, seed=3)
    mesh["skirt_mask"].zero_()
    patches, triangles = int(mesh["view"].shape[0]), int(mesh["triangles"].shape[0])
    frames = []
    for n in (patches, (1 << 25) // (6 * triangles) + 1):
        raster = TerrainRaster(WIDTH, HEIGHT, n, triangles)
        bits = raster.capacity.bit_length() + (raster.capacity * TILES).bit_length()
        assert (bits > 64) == (n > patches)
        gbuffer = raster.allocate_gbuffer(3)
        for _ in range(2):  # a second frame starts from the first one's counters
            raster.render(mesh, 0.5, tf, gbuffer)
        torch.cuda.synchronize()
        frames.append(gbuffer)
        raster.close()
    small, large = frames
    assert (small["surface_id"] >= 0).sum() > WIDTH * HEIGHT // 10
    # emission order differs from frame to frame: a pixel whose nearest triangles tie in depth may take either
    assert torch.equal(small["depth"], large["depth"])
    same = (small["position"] == large["position"]).all(-1) & (small["cell_id"] == large["cell_id"])
    assert float((~same).float().mean()) <= 1e-5
