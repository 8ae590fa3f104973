"""Triangles over many scheduling tiles are binned by whole warps from the wide
queue, in segments of 128 tiles: frames against the oracle with triangles just
below and above 32 tiles (the queue's limit), at segment remainders, clipped
ones (binned by the clipper), and with more segments than the queue holds (the
rest is binned by single threads). Visibility must be equal, colour within
1/255 as everywhere."""
import numpy as np
import pytest

import oracle
import scenes
import swr

pytestmark = pytest.mark.gpu


def quads_scene(sizes):
    """Quads facing the camera, front to back, quad i with sides sizes[i]."""
    rng = np.random.default_rng(2)
    P, UV, F = scenes.grid(1, 1)
    meshes, nodes, mats = [], [], []
    for i, (sx, sy) in enumerate(sizes):
        mats.append({"metallic": float(rng.random()), "roughness": float(rng.random()), "base_color": (0, 0, 0)})
        meshes.append([{"positions": P, "normals": None, "texcoords": UV, "indices": F, "material": i}])
        m = np.eye(4, dtype=np.float32)
        m[0, 0], m[1, 1] = sx, sy
        m[:3, 3] = (0.004 * (i % 7), -0.003 * (i % 5), -0.01 * i)
        w = m.T.reshape(16).copy()
        nodes.append({"world": w, "local": w, "mesh": i})
    return {"meshes": meshes, "nodes": nodes, "materials": mats, "textures": [scenes.noise_texture(rng, 32)],
            "cubemap": scenes.cubemap_faces(rng, 8), "cubemap_face_size": 8, "voxel_grid_size": 16,
            "specular_samples": 8, "brdf_lut_size": 16}


def check(sizes, w, h, tile, dist=3.0):
    s = swr.Scene(quads_scene(sizes))
    cam = swr.make_camera((0.0, 0.0, dist), (0.0, 0.0, 0.0), 1.0, w, h, 40.0)
    r = swr.Renderer(w, h, sched_tile=tile)
    for _ in range(2):  # the second frame starts from the first one's queue
        r.render(s, cam)
        rgba, vis = r.blit(), r.visbuffer()
    orgba, ovis, _, _ = oracle.render(s, cam, w, h, rsqrt_mode=swr.RSQRT_AARCH64, threads=1)
    assert np.array_equal(vis, ovis)
    d = np.abs(rgba[:h & ~1].view(np.uint8).astype(np.int32) - orgba[:h & ~1].view(np.uint8).astype(np.int32))
    assert d.max() <= 1
    pairs = r.stats().bin_pairs
    r.close()
    s.close()
    return pairs


@pytest.mark.parametrize("tile,w,h", [(8, 200, 120), (16, 333, 257), (32, 500, 300), (64, 900, 700)])
def test_edges_of_the_queue(tile, w, h):
    # At 3 units a unit is h / 3.28 px: sides that cross 4x8 = 32 tiles and
    # whole segments, then quads past the screen's edges (clipped).
    px = 3.28 / h
    sizes = [((a * tile + b) * px, (c * tile + b) * px)
             for a, c in ((3, 7), (4, 7), (7, 3), (31, 0.5), (32, 0.5), (15, 7), (16, 8)) for b in (-9, -1, 0, 1, 9)]
    check([(max(x, 0.01), max(y, 0.01)) for x, y in sizes] + [(9.0, 9.0), (12.0, 0.4), (0.4, 12.0)], w, h, tile)


@pytest.mark.parametrize("side", [2.9, 5.0])
def test_full_queue(side):
    # 2.9: inside the screen (k_frontend's half of the queue overflows); 5.0: clipped (the clipper's half).
    n = 120
    segments = check([(side, side)] * n, 1536, 1536, 8, dist=3.0) / 128
    assert segments > 32768
