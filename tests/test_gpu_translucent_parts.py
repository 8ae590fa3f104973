"""The translucent pass sorts the packets that reach each 16x16-px part of a
scheduling tile: by rank up to 256 of them, by bitonic passes above. Stacks of
glass quads on both sides of that line, at every scheduling tile, an odd size
and both reciprocal square roots, with and without baked light, against the
oracle (colour within 1/255, visibility equal)."""
import numpy as np
import pytest

import oracle
import scenes
import swr

pytestmark = pytest.mark.gpu


def glass_stack(n):
    rng = np.random.default_rng(n)
    P, UV, F = scenes.grid(1, 1)
    meshes, nodes, mats = [], [], []
    for i in range(n):
        glass = i != n // 2  # one opaque quad in the middle of the stack
        mats.append({"metallic": float(rng.random()), "roughness": float(rng.random()), "base_color": (0, 0, 0),
                     "has_transmission": 1 if glass else 0, "transmission": float(rng.uniform(0.7, 0.99))})
        meshes.append([{"positions": P, "normals": None, "texcoords": UV, "indices": F, "material": i}])
        m = np.eye(4, dtype=np.float32)
        m[0, 0], m[1, 1] = rng.uniform(0.4, 2.5, 2)
        m[:3, 3] = (rng.uniform(-0.6, 0.6), rng.uniform(-0.6, 0.6), -0.006 * (i // 2))  # pairs tie in depth
        w = m.T.reshape(16).copy()
        nodes.append({"world": w, "local": w, "mesh": i})
    return {"meshes": meshes, "nodes": nodes, "materials": mats, "textures": [scenes.noise_texture(rng, 32)],
            "cubemap": scenes.cubemap_faces(rng, 8), "cubemap_face_size": 8, "voxel_grid_size": 12,
            "specular_samples": 8, "brdf_lut_size": 16}


@pytest.mark.parametrize("n,gi", [(5, True), (128, False), (200, False), (420, True)])
@pytest.mark.parametrize("mode", [swr.RSQRT_AARCH64, swr.RSQRT_IEEE])
def test_glass_stack(n, gi, mode):
    sd = glass_stack(n)
    s = swr.Scene(sd, gi=gi)
    w, h = 83, 70
    cam = swr.make_camera((0.0, 0.0, 2.2), (0.0, 0.0, 0.0), 1.0, w, h, 40.0)
    orgba, ovis, _, _ = oracle.render(s, cam, w, h, rsqrt_mode=mode, threads=1)
    for tile in (8, 16, 32, 64):
        r = swr.Renderer(w, h, rsqrt_mode=mode, sched_tile=tile)
        r.render(s, cam)
        rgba, vis = r.blit(), r.visbuffer()
        r.close()
        assert np.array_equal(vis, ovis), tile
        d = np.abs(rgba[:h & ~1].view(np.uint8).astype(np.int32) - orgba[:h & ~1].view(np.uint8).astype(np.int32))
        assert d.max() <= 1, (tile, d.max())
    s.close()
