"""A frame's counts and kernel forms. Set-up triangles and (triangle, tile)
pairs count every triangle that the reference bins, and the triangles left out
of the bins are exactly those the oracle finds by integer edge tests to hold no
pixel centre, up to the 2^24 bound of that claim. The raster and the shading
take their other CTA shapes, and 16-px tiles their culling form, at the stated
numbers of tiles per SM, triangles per tile and pixels per SM of this device,
with the same frame on both sides."""
import numpy as np
import pytest

import oracle
import scenes
import swr
from test_gpu_parity import tie_across_rounds_scene
from test_gpu_unsampled import specks_scene

pytestmark = pytest.mark.gpu
SIZES = [0.11, 0.25, 0.5, 0.5625, 0.8, 1.0, 1.0625, 1.5, 2.0, 2.3, 3.0, 4.0]


@pytest.mark.parametrize("jitter", [0.0, 1.0])
@pytest.mark.parametrize("w,h", [(333, 64), (3840, 128), (20000, 64)])
def test_counts(w, h, jitter):
    s = swr.Scene(specks_scene(SIZES, w, h, jitter, seed=w + int(10 * jitter)))
    cam = swr.make_camera((0.0, 0.0, 1.0), (0.0, 0.0, 0.0), 1.0, w, h, 10.0)
    _, ovis, _, res = oracle.render(s, cam, w, h, rsqrt_mode=swr.RSQRT_AARCH64, threads=1, counts=True)
    assert 0 < res.unsampled < res.setup
    for i, tile in enumerate((8, 16, 32, 64)):
        r = swr.Renderer(w, h, sched_tile=tile)
        r.render(s, cam)
        assert np.array_equal(r.visbuffer(), ovis), tile
        st, d = r.stats(), r.detail()
        assert (st.setup_triangles, st.bin_pairs) == (res.setup, res.pairs[i]), tile
        assert (d.unsampled_triangles, d.unsampled_pairs) == (res.unsampled, res.unsampled_pairs[i]), tile
        r.close()
    s.close()


def sms():
    return pytest.importorskip("torch").cuda.get_device_properties(0).multi_processor_count


def frame(s, w, h, tile):
    pos, at, fov, w, h, far = scenes.default_camera_params(s.info(), w, h)
    r = swr.Renderer(w, h, sched_tile=tile)
    r.render(s, swr.make_camera(pos, at, fov, w, h, far))
    out = r.blit(), r.visbuffer(), r.detail()
    r.close()
    return out


@pytest.mark.parametrize("below", [0, 1])
def test_crowded_tiles_take_the_narrow_raster(below):
    """12 tiles of 32 px per SM: the raster's CTAs are narrow from 176 triangles a tile on."""
    n = sms()
    count = -(-176 * 12 * n // 20480) - below
    s = swr.Scene(scenes.spheres_scene(seed=8, count=count, subdiv=5, tex_size=16, cube_size=16, voxel=16))
    rgba, vis, d = frame(s, 64 * n - 3, 64 * 3 - 1, 32)
    assert d.raster_threads == (256 if below else 128)
    want_rgba, want_vis, _ = frame(s, 64 * n - 3, 64 * 3 - 1, 8)
    assert np.array_equal(vis, want_vis) and np.array_equal(rgba[:190], want_rgba[:190])
    s.close()


@pytest.mark.parametrize("extra", [-1, 1])
def test_culling_with_many_32px_tiles(extra):
    """24 tiles a view, on both sides of the number of tiles from which the raster's CTAs are narrow; bins of several
    rounds of either width, with a tie that the last of the tied triangles wins."""
    s = swr.Scene(tie_across_rounds_scene(300))
    w, h = 190, 127
    cam = swr.make_camera((0.0, 0.0, 3.0), (0.0, 0.0, 0.0), 1.0, w, h, 40.0)
    _, ovis, _, _ = oracle.render(s, cam, w, h, rsqrt_mode=swr.RSQRT_AARCH64, threads=1)
    views = 44 * sms() // 24 + extra
    b = swr.Batch(sched_tile=32)
    b.render(swr.Batch.views([(s, cam, w, h, 2.0, swr.RSQRT_AARCH64)] * views))
    for i in range(views):
        assert np.array_equal(b.output(i, w, h)[1], ovis), i
    b.close()
    s.close()


@pytest.fixture(scope="module")
def spheres():
    s = swr.Scene(scenes.spheres_scene(seed=8, count=20, subdiv=3, tex_size=16, cube_size=16, voxel=16))  # 25,600
    yield s
    s.close()


# Sizes in 64-px tiles, n SMs; a form, and whether it is taken there.
def forms(n):
    return {"wide shading below": ((n - 1) // 8, 8, 64, "shade_threads", 128),
            "wide shading": (-(-n // 8), 8, 64, "shade_threads", 1024),
            "narrow raster below": (n - 1, 11, 32, "raster_threads", 256),
            "narrow raster": (n, 11, 32, "raster_threads", 128),
            "16-px culling below": (13, 2, 16, "culling", 0), "16-px culling": (5, 5, 16, "culling", 1)}


@pytest.mark.parametrize("name", list(forms(16)))
def test_forms(spheres, name):
    cols, rows, tile, field, value = forms(sms())[name]
    w, h = 64 * cols - 3, 64 * rows - 1
    rgba, vis, d = frame(spheres, w, h, tile)
    assert getattr(d, field) == value
    want_rgba, want_vis, plain = frame(spheres, w, h, 8)
    assert (plain.raster_threads, plain.shade_threads, plain.culling) == (128, 0, 0)
    assert np.array_equal(vis, want_vis) and np.array_equal(rgba[:h & ~1], want_rgba[:h & ~1])
    assert (vis != np.uint64(2 ** 64 - 1)).sum() > 1000
