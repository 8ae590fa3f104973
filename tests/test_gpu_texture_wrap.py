"""Texture addressing on the device: repeat over power-of-two sizes is a
conversion and a mask, everything else the general form. Textures with
power-of-two, odd and mixed sizes, every pair of wrap modes and texture
coordinates far outside [0, 1] (past 2^31 texels too), against the oracle:
visibility equal, colour within 1/255."""
import numpy as np
import pytest

import oracle
import scenes
import swr

pytestmark = pytest.mark.gpu


def wrap_scene(tw, th, scale, shift):
    rng = np.random.default_rng(tw * 131 + th)
    rgb = rng.random((th, tw, 3), dtype=np.float32)
    tex = {"width": tw, "height": th, "type": scenes.TEX_SRGB, "rgba8": scenes.pack_rgba8(rgb)}
    P, UV, F = scenes.grid(3, 3)
    UV = (UV * np.float32(scale) + np.float32(shift)).astype(np.float32)
    meshes, nodes, mats = [], [], []
    for i in range(9):
        mats.append({"metallic": 0.1, "roughness": 0.8, "base_color": (0, i % 3, i // 3)})
        meshes.append([{"positions": P, "normals": None, "texcoords": UV, "indices": F, "material": i}])
        m = np.eye(4, dtype=np.float32)
        m[:3, 3] = (1.02 * (i % 3 - 1), 1.02 * (i // 3 - 1), 0.0)
        w = m.T.reshape(16).copy()
        nodes.append({"world": w, "local": w, "mesh": i})
    return {"meshes": meshes, "nodes": nodes, "materials": mats, "textures": [tex],
            "cubemap": scenes.cubemap_faces(rng, 8), "cubemap_face_size": 8, "voxel_grid_size": 8,
            "specular_samples": 4, "brdf_lut_size": 8}


@pytest.mark.parametrize("tw,th", [(64, 64), (1, 16), (48, 20), (64, 20), (20, 64)])
@pytest.mark.parametrize("scale,shift", [(1.0, 0.0), (3.0, -7.25), (5.0, 1.0e6), (8.0, -1.0e8), (64.0, 6.0e8)])
def test_wrap(tw, th, scale, shift):
    s = swr.Scene(wrap_scene(tw, th, scale, shift))
    w, h = 160, 160
    cam = swr.make_camera((0.0, 0.0, 3.2), (0.0, 0.0, 0.0), 1.0, w, h, 10.0)
    orgba, ovis, _, _ = oracle.render(s, cam, w, h, rsqrt_mode=swr.RSQRT_AARCH64, threads=1)
    r = swr.Renderer(w, h, sched_tile=32)
    r.render(s, cam)
    rgba, vis = r.blit(), r.visbuffer()
    r.close()
    s.close()
    assert np.array_equal(vis, ovis)
    d = np.abs(rgba.view(np.uint8).astype(np.int32) - orgba.view(np.uint8).astype(np.int32))
    assert d.max() <= 1
