"""Shading skips the sunlight of pixels turned away from the sun or in shadow,
where the material's base colour is bounded; elsewhere the terms are formed as
always (0 times an infinite factor is not 0). Spheres lit from the side, with
factors on both sides of the bound, against the oracle."""
import numpy as np
import pytest

import oracle
import scenes
import swr

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("factor", [0.8, 0.0, -2.0, 1.0e6, 1.1e6, 1.0e30, float("inf"), float("nan")])
@pytest.mark.parametrize("mode", [swr.RSQRT_AARCH64, swr.RSQRT_IEEE])
def test_unlit_pixels(factor, mode):
    sd = scenes.small_scene(seed=9, count=5)
    for i, m in enumerate(sd["materials"]):
        m["base_color_factor"] = (factor, 0.5, factor if i % 2 else 0.25, 1.0)
    s = swr.Scene(sd)
    w, h = 200, 144
    cam = swr.make_camera(*scenes.default_camera_params(s.info(), w, h))
    orgba, ovis, _, _ = oracle.render(s, cam, w, h, rsqrt_mode=mode, threads=1)
    for tile in (16, 64):  # shaded in the raster kernel, and apart
        r = swr.Renderer(w, h, rsqrt_mode=mode, sched_tile=tile)
        r.render(s, cam)
        rgba, vis = r.blit(), r.visbuffer()
        r.close()
        assert np.array_equal(vis, ovis)
        d = np.abs(rgba.view(np.uint8).astype(np.int32) - orgba.view(np.uint8).astype(np.int32))
        assert d.max() <= 1
    s.close()
