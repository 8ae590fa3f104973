"""Occlusion culling in 16- and 32-px scheduling tiles: bins of more than one round (a
packet per thread of the CTA) are culled against the depths of earlier rounds,
lighter ones are not. Stacks of screen-filling quads with a tie that arrives
last, with bins on both sides of the line, shaded apart and in the raster
kernel, against the oracle: visibility must be equal and the last of the tied
quads must win."""
import numpy as np
import pytest

import oracle
import swr
from test_gpu_parity import tie_across_rounds_scene

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [40, 110, 130, 300])
@pytest.mark.parametrize("fused", [False, True])
def test_ties_and_culling_in_32px_tiles(n, fused):
    s = swr.Scene(tie_across_rounds_scene(n))
    w, h = 190, 127
    cam = swr.make_camera((0.0, 0.0, 3.0), (0.0, 0.0, 0.0), 1.0, w, h, 40.0)
    orgba, ovis, _, _ = oracle.render(s, cam, w, h, rsqrt_mode=swr.RSQRT_AARCH64, threads=1)
    b = swr.Batch(sched_tile=32, fused_shade=fused)
    b.render(swr.Batch.views([(s, cam, w, h, 2.0, swr.RSQRT_AARCH64)] * 2))
    for i in range(2):
        rgba, vis = b.output(i, w, h)
        assert np.array_equal(vis, ovis)
        d = np.abs(rgba[:h & ~1].view(np.uint8).astype(np.int32) - orgba[:h & ~1].view(np.uint8).astype(np.int32))
        assert d.max() <= 1
    b.close()
    r = swr.Renderer(w, h, sched_tile=32)
    r.render(s, cam)
    assert np.array_equal(r.visbuffer(), ovis)
    if n in (40, 300):
        assert (r.stats().culled_pairs > 0) == (n == 300)
    r.close()
    s.close()


@pytest.mark.parametrize("views,cap", [(75, 0), (77, 0), (77, 3)])
def test_many_32px_tiles(views, cap):
    """24 tiles a view: 12 tiles per SM of 152 lie between 75 and 77 views, where
    the raster's CTA width changes; every view must equal the oracle's."""
    s = swr.Scene(tie_across_rounds_scene(300))
    w, h = 190, 127
    cam = swr.make_camera((0.0, 0.0, 3.0), (0.0, 0.0, 0.0), 1.0, w, h, 40.0)
    _, ovis, _, _ = oracle.render(s, cam, w, h, rsqrt_mode=swr.RSQRT_AARCH64, threads=1)
    b = swr.Batch(sched_tile=32, raster_ctas_per_sm=cap)
    b.render(swr.Batch.views([(s, cam, w, h, 2.0, swr.RSQRT_AARCH64)] * views))
    for i in range(views):
        assert np.array_equal(b.output(i, w, h)[1], ovis)
    b.close()
    s.close()


@pytest.mark.parametrize("n", [480, 520, 1000])
@pytest.mark.parametrize("gi", [False, True])
def test_ties_and_culling_in_16px_tiles(n, gi):
    """16 tiles of 16 px: from 1,024 triangles on they are culled."""
    s = swr.Scene(tie_across_rounds_scene(n), gi=gi)
    w, h = 61, 45
    cam = swr.make_camera((0.0, 0.0, 3.0), (0.0, 0.0, 0.0), 1.0, w, h, 40.0)
    for mode in (swr.RSQRT_AARCH64, swr.RSQRT_IEEE):
        orgba, ovis, _, _ = oracle.render(s, cam, w, h, rsqrt_mode=mode, threads=1)
        r = swr.Renderer(w, h, rsqrt_mode=mode, sched_tile=16)
        r.render(s, cam)
        assert np.array_equal(r.visbuffer(), ovis)
        rgba = r.blit()
        d = np.abs(rgba[:h & ~1].view(np.uint8).astype(np.int32) - orgba[:h & ~1].view(np.uint8).astype(np.int32))
        assert d.max() <= 1
        assert (r.stats().culled_pairs > 0) == (n > 500)
        r.close()
    s.close()
