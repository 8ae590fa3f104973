"""The allocation-free frame takes 65,536 (triangle, 64-px tile) pairs and no
more, whatever tiles it rasterizes on: frames at the limit equal the regular
ones, frames one pair past it return SWR_OVERFLOW. Triangles over the whole
picture, triangles without a pixel centre (they count), and triangles cut by
the frustum into fans, whose pairs a renderer with 64-px tiles counts."""
import ctypes as C

import numpy as np
import pytest

import scenes
import swr

pytestmark = pytest.mark.gpu
SIZE, LIMIT = 512, 65536
FULL = [(5, 5), (5, 507), (507, 5)]               # touches all 64 tiles of 64 px
SPECK = [(100.1, 100.1), (100.1, 100.3), (100.3, 100.1)]  # one tile, no pixel centre
CUT = [(-60, 20), (500, 40), (480, 500)]          # crosses the left edge: two fan triangles


def scene_of(triangles):
    """Triangles in pixels of a 512x512 picture seen from distance 1, each in both windings."""
    unit = 2.0 * np.tan(0.5) / SIZE
    P = []
    for i, t in enumerate(triangles):
        for w in (t, t[::-1]):
            P += [[(x - SIZE / 2) * unit, (SIZE / 2 - y) * unit, -1e-6 * i] for x, y in w]
    rng = np.random.default_rng(3)
    eye = np.eye(4, dtype=np.float32).reshape(16)
    return {"meshes": [[{"positions": np.array(P, np.float32), "normals": None,
                         "texcoords": np.zeros((len(P), 2), np.float32), "indices": np.arange(len(P), dtype=np.uint32),
                         "material": 0}]],
            "nodes": [{"world": eye, "local": eye, "mesh": 0}], "materials": [{"metallic": 0.2, "roughness": 0.6}],
            "textures": [scenes.noise_texture(rng, 8)], "cubemap": scenes.cubemap_faces(rng, 8), "cubemap_face_size": 8,
            "voxel_grid_size": 8, "specular_samples": 4, "brdf_lut_size": 8}


def render(triangles):
    """Pairs that a renderer counts, the allocation-free frame's status, and whether it equals the renderer's frame."""
    torch = pytest.importorskip("torch")
    s = swr.Scene(scene_of(triangles))
    cam = swr.make_camera((0.0, 0.0, 1.0), (0.0, 0.0, 0.0), 1.0, SIZE, SIZE, 10.0)
    r = swr.Renderer(SIZE, SIZE, sched_tile=64)
    r.render(s, cam)
    want = r.blit(), r.visbuffer()
    pairs = r.stats().bin_pairs
    r.close()
    rgba = torch.zeros(SIZE, SIZE, dtype=torch.int32, device="cuda")
    vis = torch.zeros(SIZE, SIZE, dtype=torch.int64, device="cuda")
    st = swr.lib().swr_render_frame_noalloc(s.handle, C.byref(cam), SIZE, SIZE, 2.0, swr.RSQRT_AARCH64,
                                            C.c_void_p(rgba.data_ptr()), C.c_void_p(vis.data_ptr()), None)
    same = np.array_equal(rgba.cpu().numpy().view(np.uint32), want[0]) and \
        np.array_equal(vis.cpu().numpy().view(np.uint64), want[1])
    s.close()
    return pairs, st, same


@pytest.mark.parametrize("full,specks", [(1024, 0), (1023, 64)])
def test_at_and_past_the_limit(full, specks):
    assert render([FULL] * full + [SPECK] * specks) == (LIMIT, swr.SWR_OK, True)
    pairs, st, _ = render([FULL] * full + [SPECK] * (specks + 1))
    assert (pairs, st) == (LIMIT + 1, swr.SWR_OVERFLOW)


def test_limit_counts_fans():
    one, st, same = render([CUT])
    assert one > 40 and st == swr.SWR_OK and same
    n, rest = divmod(LIMIT, one)
    assert render([CUT] * n + [SPECK] * rest) == (LIMIT, swr.SWR_OK, True)
    pairs, st, _ = render([CUT] * n + [SPECK] * (rest + 1))
    assert (pairs, st) == (LIMIT + 1, swr.SWR_OVERFLOW)
