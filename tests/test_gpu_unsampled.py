"""Triangles whose bounding box holds at most 2x2 pixel centres, none of them
inside, are not binned. Meshes of triangles from far below to a few pixels, in
regular rows whose edges run through pixel centres and in jittered ones, at
frame widths on both sides of the 2^24 bound of the claim: visibility must equal
the oracle's, and the counts of set-up triangles and (triangle, tile) pairs
those of a frame whose triangles are all binned (the allocation-free entry
point's limits need them all, so its frames bin them)."""
import numpy as np
import pytest

import oracle
import scenes
import swr

pytestmark = pytest.mark.gpu


def specks_scene(px_sizes, w, h, jitter, seed):
    """One grid per size, its cells `size` pixels wide for a camera at z = 1
    with a vertical field of 1 radian; cells sit on subpixel sixteenths unless
    jittered, so edges and vertices meet pixel centres exactly."""
    rng = np.random.default_rng(seed)
    unit = 2.0 * np.tan(0.5) / h  # world units per pixel at distance 1
    meshes, nodes = [], []
    for i, px in enumerate(px_sizes):
        n = 40
        P, UV, F = scenes.grid(n, n)
        P = P.copy() * np.float32(n * px * unit)
        if jitter:
            P += rng.uniform(-0.4, 0.4, P.shape).astype(np.float32) * np.float32(px * unit * jitter)
        cx = (i + 0.5) / len(px_sizes) - 0.5
        P[:, 0] += np.float32(cx * w * unit)
        meshes.append([{"positions": P.astype(np.float32), "normals": None, "texcoords": UV, "indices": F,
                        "material": 0}])
        eye = np.eye(4, dtype=np.float32).reshape(16)
        nodes.append({"world": eye, "local": eye, "mesh": i})
    return {"meshes": meshes, "nodes": nodes, "materials": [{"metallic": 0.3, "roughness": 0.6}],
            "textures": [scenes.noise_texture(rng, 8)], "cubemap": scenes.cubemap_faces(rng, 8),
            "cubemap_face_size": 8, "voxel_grid_size": 8, "specular_samples": 4, "brdf_lut_size": 8}


@pytest.mark.parametrize("jitter", [0.0, 0.3, 1.0])
@pytest.mark.parametrize("w,h", [(333, 64), (3840, 128), (9000, 80), (20000, 64)])
def test_specks(w, h, jitter):
    sizes = [0.11, 0.25, 0.5, 0.5625, 0.8, 1.0, 1.0625, 1.5, 2.0, 2.3, 3.0, 4.0]
    s = swr.Scene(specks_scene(sizes, w, h, jitter, seed=w + int(10 * jitter)))
    cam = swr.make_camera((0.0, 0.0, 1.0), (0.0, 0.0, 0.0), 1.0, w, h, 10.0)
    _, ovis, _, _ = oracle.render(s, cam, w, h, rsqrt_mode=swr.RSQRT_AARCH64, threads=1)
    assert (ovis != np.uint64(2 ** 64 - 1)).sum() > 1000
    for tile in (16, 64):
        r = swr.Renderer(w, h, sched_tile=tile)
        r.render(s, cam)
        assert np.array_equal(r.visbuffer(), ovis), tile
        st = r.stats()
        assert st.setup_triangles <= st.bin_pairs
        r.close()
    s.close()
