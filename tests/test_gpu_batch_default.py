"""The form a batch of several views takes by itself: 32-px tiles shaded in the
raster kernel for small views, shaded apart for larger ones and for scenes of
many triangles; 16-px tiles for few. Either form gives the frames of
a renderer."""
import numpy as np
import pytest

import scenes
import swr

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def made():
    s = {"light": swr.Scene(scenes.small_scene(seed=4)),  # 1,920 triangles
         "heavy": swr.Scene(scenes.spheres_scene(seed=4, count=79, subdiv=3, tex_size=16, cube_size=16, voxel=16)),
         "below": swr.Scene(scenes.spheres_scene(seed=4, count=78, subdiv=3, tex_size=16, cube_size=16, voxel=16))}
    yield s
    for x in s.values():
        x.close()


# Scene, size and number of views; tile and form. 48 tiles of 64 px a view is
# 8x6; the scenes have 1,920, 101,120 and 99,840 triangles.
CASES = [("light", 512, 384, 40, 32, 1), ("light", 513, 384, 40, 32, 0), ("light", 320, 240, 100, 32, 1),
         ("heavy", 512, 384, 40, 32, 0), ("below", 512, 384, 40, 32, 1), ("light", 512, 384, 2, 16, 0),
         ("light", 1920, 1080, 2, 32, 0)]


@pytest.mark.parametrize("scene,w,h,n,tile,fused", CASES)
def test_default_form(made, scene, w, h, n, tile, fused):
    s = made[scene]
    cams = []
    for i in range(n):
        pos, at, fov, _, _, far = scenes.default_camera_params(s.info(), w, h)
        cams.append(swr.make_camera((pos[0] + 0.02 * i, pos[1], pos[2]), at, fov, w, h, far))
    b = swr.Batch()
    views = swr.Batch.views([(s, c, w, h, 2.0, swr.RSQRT_AARCH64) for c in cams])
    t = b.tuning(views)
    assert (t["tuned"], t["sched_tile"], t["fused_shade"]) == (0, tile, fused)
    b.render(views)
    b.sync()
    r = swr.Renderer(w, h)
    for i in {0, n // 2, n - 1}:
        r.render(s, cams[i])
        want_rgba, want_vis = r.blit(), r.visbuffer()
        rgba, vis = b.output(i, w, h)
        assert np.array_equal(vis, want_vis) and np.array_equal(rgba[:h & ~1], want_rgba[:h & ~1]), i
    r.close()
    b.close()
