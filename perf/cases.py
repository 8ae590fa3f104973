"""Performance cases: the calls a program makes into this library, with the
sizes and options of real use.

The library is a per-frame renderer with a batched and a served form and a
scene loader, so a case is one frame of one of them (or one scene load)
through the binding's public classes. Scenes are the seeded synthetic ones of
scenes.py (spheres; displaced grids and icospheres with log-uniform triangle
sizes; glass; every texture slot), textures are seeded value noise made on the
GPU, cameras are drawn from the seed. Every output is whole: RGBA8 frames,
visibility buffers, the tables of a loaded scene.
"""
import ctypes as C
import math
import os
import random
import sys

import numpy as np
import torch

_ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, os.path.join(_ROOT, "swraster-viewer_gb300"))
import scenes  # noqa: E402
import swr  # noqa: E402

# Resolutions of batched views and served requests, cycled over the views.
VIEW_SIZES = [(320, 240), (640, 480), (1280, 720), (1920, 1080)]
SCENE_SIZES = [(640, 480), (960, 540), (1280, 720), (1600, 900), (1920, 1080), (2560, 1440)]


def listed():
    return [
        # A preview: few objects in a small picture, where the fixed cost of
        # a frame is all there is.
        _frame("frame_preview", "spheres", 6, 2, 320, 240),
        # The 81,920-triangle sphere scene in a 1280x720 window.
        _frame("frame_720p", "spheres", 64, 3, 1280, 720),
        # The headline: 2M triangles at 4K, eight 2048^2 textures.
        _stress("frame_4k", 2_000_000, 3840, 2160, textures=8, tex=2048),
        # Materials with every texture slot (normal maps, metallic-roughness,
        # emissive, occlusion), on a host without the Arm estimate.
        _stress("frame_materials", 400_000, 1920, 1080, textures=4, tex=1024, slots=True, ieee=True),
        # The interactive loop: automatic exposure between frames, a window
        # of an odd size.
        _stress("loop_exposure", 150_000, 1367, 769, textures=4, tex=1024, dt=1.0 / 60.0),
        # Glass: translucent spheres and planes sorted and blended per pixel.
        dict(_frame("frame_glass", "glass", 24, 3, 1600, 900), dt=1.0 / 60.0),
        # Baked voxel lighting.
        _stress("frame_baked_gi", 80_000, 1280, 720, textures=2, tex=512, gi=True),
        # 64 views of one scene in one launch sequence (thumbnails, turntables).
        {"name": "batch_views", "kind": "batch_views", "objects": 64, "subdiv": 3, "views": 64, "scale": 1.0,
         "graph": True},
        # Uneven scenes, one view each, in one launch sequence.
        {"name": "batch_scenes", "kind": "batch_scenes", "scenes": 8, "tris_min": 10_000, "tris_max": 1_500_000,
         "textures": 2, "tex": 1024, "scale": 1.0, "graph": True},
        # A burst of requests to the server over resident scenes.
        {"name": "serve_burst", "kind": "serve", "scenes": 3, "tris_min": 20_000, "tris_max": 500_000, "textures": 2,
         "tex": 1024, "requests": 24, "scale": 1.0},
        # A frame inside a program that must not allocate while rendering.
        {"name": "frame_noalloc", "kind": "noalloc", "objects": 10, "subdiv": 3, "width": 500, "height": 281},
        # Opening a scene: mip chains, environment prefilter, tangents, sun
        # visibility and the voxel light bake.
        {"name": "scene_load", "kind": "load", "objects": 12, "subdiv": 4, "tex": 1024, "cube": 128, "voxel": 64,
         "gi": True},
    ]


def _frame(name, scene, objects, subdiv, width, height, ieee=False):
    return {"name": name, "kind": "frame", "scene": scene, "objects": objects, "subdiv": subdiv, "width": width,
            "height": height, "dt": 0.0, "ieee": ieee}


def _stress(name, triangles, width, height, textures, tex, slots=False, ieee=False, dt=0.0, gi=False):
    return {"name": name, "kind": "frame", "scene": "stress", "triangles": triangles, "width": width,
            "height": height, "textures": textures, "tex": tex, "slots": slots, "ieee": ieee, "dt": dt, "gi": gi}


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng: random.Random):
    """A case of the listed ranges: any kind, sizes log-uniform."""
    kind = rng.choice(["spheres", "stress", "stress", "slots", "loop", "glass", "gi", "batch_views", "batch_scenes",
                       "serve", "noalloc", "load"])
    w = _log(rng, 200, 3840)
    h = max(64, min(2160, int(w * rng.uniform(0.5, 0.8))))
    ieee = rng.random() < 0.3
    if kind == "spheres":
        c = _frame("", "spheres", _log(rng, 6, 96), rng.randint(2, 4), min(w, 1920), min(h, 1200), ieee)
    elif kind == "stress":
        c = _stress("", _log(rng, 20_000, 1_800_000), w, h, rng.randint(1, 8), rng.choice([512, 1024]), ieee=ieee)
    elif kind == "slots":
        c = _stress("", _log(rng, 20_000, 600_000), min(w, 2560), min(h, 1440), rng.randint(1, 4),
                    rng.choice([512, 1024]), slots=True, ieee=ieee)
    elif kind == "loop":
        c = _stress("", _log(rng, 20_000, 400_000), min(w, 1920), min(h, 1080), rng.randint(1, 4), 512, ieee=ieee,
                    dt=rng.choice([1.0 / 144.0, 1.0 / 60.0, 0.1]))
    elif kind == "glass":
        c = dict(_frame("", "glass", _log(rng, 4, 32), rng.randint(2, 3), min(w, 1600), min(h, 900), ieee),
                 dt=rng.choice([0.0, 1.0 / 60.0]))
    elif kind == "gi":
        c = _stress("", _log(rng, 10_000, 100_000), min(w, 1920), min(h, 1080), rng.randint(1, 2), 512, gi=True)
    elif kind == "batch_views":
        c = {"kind": kind, "objects": _log(rng, 8, 64), "subdiv": rng.randint(2, 3), "views": _log(rng, 2, 64),
             "scale": round(rng.uniform(0.2, 1.0), 3), "graph": rng.random() < 0.7}
    elif kind == "batch_scenes":
        c = {"kind": kind, "scenes": rng.randint(2, 8), "tris_min": 10_000, "tris_max": _log(rng, 50_000, 1_200_000),
             "textures": rng.randint(1, 3), "tex": rng.choice([512, 1024]), "scale": round(rng.uniform(0.3, 1.0), 3),
             "graph": rng.random() < 0.7}
    elif kind == "serve":
        c = {"kind": kind, "scenes": rng.randint(1, 3), "tris_min": 10_000, "tris_max": _log(rng, 30_000, 500_000),
             "textures": rng.randint(1, 2), "tex": 512, "requests": rng.randint(1, 24),
             "scale": round(rng.uniform(0.3, 1.0), 3)}
    elif kind == "noalloc":
        c = {"kind": kind, "objects": rng.randint(1, 10), "subdiv": rng.randint(1, 3), "width": rng.randint(48, 512),
             "height": rng.randint(48, 300)}
    else:
        c = {"kind": "load", "objects": rng.randint(4, 12), "subdiv": rng.randint(2, 4), "tex": _log(rng, 128, 1024),
             "cube": rng.choice([32, 64, 128]), "voxel": rng.randint(24, 64), "gi": rng.random() < 0.5}
    c.pop("name", None)
    return c


# ------------------------------------------------------------------ inputs


def _noise(size, seed, channels=3):
    """Seeded value noise of a few octaves in [0, 1], (size, size, channels), made on the GPU."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    out = torch.zeros(1, channels, size, size, device="cuda")
    amp, total = 1.0, 0.0
    for cells in (8, 32, 128):
        lat = torch.rand(1, channels, cells, cells, generator=g, device="cuda")
        out += amp * torch.nn.functional.interpolate(lat, size=(size, size), mode="bilinear", align_corners=False)
        total += amp
        amp *= 0.5
    return (out / total)[0].permute(1, 2, 0).cpu().numpy()


def _texture(size, seed, kind):
    n = _noise(size, seed)
    if kind == scenes.TEX_NORMAL:
        xy = (n[..., :2] - 0.5) * 1.2
        z = np.sqrt(np.clip(1.0 - (xy * xy).sum(-1), 0.05, 1.0))
        v = np.concatenate([xy, z[..., None]], -1)
        n = v / np.linalg.norm(v, axis=-1, keepdims=True) * 0.5 + 0.5
    elif kind == scenes.TEX_LINEAR:
        n = 0.3 + 0.7 * n
    return {"width": size, "height": size, "type": kind, "rgba8": scenes.pack_rgba8(n)}


def _big_textures(sd, seed, size):
    """The scene's textures replaced by ones of `size` of the same kind."""
    sd["textures"] = [_texture(size, seed * 101 + i, t["type"]) for i, t in enumerate(sd["textures"])]
    return sd


def _stress_scene(seed, triangles, w, h, textures, tex, slots=False, voxel=128):
    sd, cam = scenes.stress_scene(seed=seed, triangles=triangles, width=w, height=h, n_textures=textures, tex_size=16,
                                  voxel=voxel, all_slots=slots)
    return _big_textures(sd, seed, tex), cam


def _scene_sizes(case):
    n = case["scenes"]
    lo, hi = case["tris_min"], case["tris_max"]
    tris = [int(lo * (hi / lo) ** (i / max(1, n - 1))) for i in range(n)] if n > 1 else [hi]
    return tris


def _scaled(size, scale):
    return max(16, int(size[0] * scale)), max(16, int(size[1] * scale))


def _view_sizes(case, table):
    n = case.get("views") or case.get("requests") or case["scenes"]
    return [_scaled(table[i % len(table)], case["scale"]) for i in range(n)]


class _Device:
    """A device pointer of the library as an array other libraries can view; it holds the handle that owns it."""

    def __init__(self, ptr, shape, typestr, owner):
        self.owner = owner
        self.__cuda_array_interface__ = {"shape": shape, "typestr": typestr, "data": (ptr, False), "version": 3}


def _view_of(ptr, shape, typestr, owner):
    return torch.as_tensor(_Device(ptr, shape, typestr, owner), device="cuda")


def _host_view(ptr, count, dtype, owner):
    """`count` values at a host pointer of the library as an array that holds the handle that owns them."""
    dtype = np.dtype(dtype)
    buf = (C.c_uint8 * (count * dtype.itemsize)).from_address(C.cast(ptr, C.c_void_p).value)
    buf.owner = owner
    return np.frombuffer(buf, dtype)


def _orbit(rng, info, w, h, *radius):
    """Parameters of a camera that orbits the scene and sees its centre. swr_camera_init takes the pitch of the given
    direction and swr_camera_update turns by it the other way (as the reference's camera does), so the target's height
    is mirrored about the camera's."""
    pos, at, fov, w, h, far = scenes.sphere_camera(rng, info, w, h, *radius)
    return pos, (at[0], 2.0 * pos[1] - at[1], at[2]), fov, w, h, far


def _frame_scene(case, seed):
    rng = np.random.default_rng(seed)
    w, h = case["width"], case["height"]
    if case["scene"] == "spheres":
        s = swr.Scene(scenes.spheres_scene(seed=seed, count=case["objects"], subdiv=case["subdiv"]))
        cam = _orbit(rng, s.info(), w, h)
    elif case["scene"] == "glass":
        sd = scenes.translucent_scene(seed=seed, count=case["objects"], subdiv=case["subdiv"], box=6.0, tex_size=256,
                                      cube_size=64)
        s = swr.Scene(sd)
        d = s.info().bounds_diagonal
        cam = _orbit(rng, s.info(), w, h, 0.6 * d, 0.9 * d)
    else:
        sd, cam = _stress_scene(seed, case["triangles"], w, h, case["textures"], case["tex"], case["slots"],
                                voxel=32 if case["gi"] else 128)
        s = swr.Scene(sd, gi=case["gi"])
    return s, swr.make_camera(*cam)


def prepare(case, seed):
    seed = int(seed) % (1 << 30)
    rng = np.random.default_rng(seed)
    kind = case["kind"]
    if kind == "frame":
        w, h = case["width"], case["height"]
        scene, cam = _frame_scene(case, seed)
        r = swr.Renderer(w, h, rsqrt_mode=swr.RSQRT_IEEE if case["ieee"] else swr.RSQRT_AARCH64)
        frame = torch.zeros(h, w, dtype=torch.int32, pin_memory=True)
        pixels = frame.numpy().view(np.uint32)
        r.set_blit_target(frame.data_ptr(), w, keep=frame)
        vis = _view_of(r.device_outputs()[1], (h, w), "<i8", r)
        return {"case": case, "scene": scene, "cam": cam, "r": r, "frame": frame, "pixels": pixels, "vis": vis}
    if kind in ("batch_views", "batch_scenes"):
        if kind == "batch_views":
            s = swr.Scene(scenes.spheres_scene(seed=seed, count=case["objects"], subdiv=case["subdiv"]))
            sizes = _view_sizes(case, VIEW_SIZES)
            items = [(s, swr.make_camera(*_orbit(rng, s.info(), w, h)), w, h) for w, h in sizes]
        else:
            sizes = _view_sizes(case, SCENE_SIZES)
            items = []
            for i, (t, (w, h)) in enumerate(zip(_scene_sizes(case), sizes)):
                sd, cam = _stress_scene(seed * 16 + i, t, w, h, case["textures"], case["tex"], voxel=64)
                items.append((swr.Scene(sd), swr.make_camera(*cam), w, h))
        px = sum(w * h for w, h in sizes)
        rgba = torch.zeros(px, dtype=torch.int32, device="cuda")
        vis = torch.zeros(px, dtype=torch.int64, device="cuda")
        views = swr.Batch.views([(s, cam, w, h, 2.0, swr.RSQRT_AARCH64) for s, cam, w, h in items])
        at = 0
        for v, (w, h) in zip(views, sizes):
            v.rgba8, v.vis = rgba.data_ptr() + 4 * at, vis.data_ptr() + 8 * at
            at += w * h
        return {"case": case, "items": items, "batch": swr.Batch(use_graph=case["graph"]), "views": views,
                "rgba": rgba, "vis": vis}
    if kind == "serve":
        srv = swr.Server(memory_budget=40 << 30, max_batch_views=64, inflight=3, use_graph=True)
        resident, requests = [], []
        for i, t in enumerate(_scene_sizes(case)):
            sd, _ = _stress_scene(seed * 16 + i, t, 1280, 720, case["textures"], case["tex"], voxel=64)
            resident.append(swr.Scene(sd))
        ids = [srv.add_scene(s) for s in resident]
        for i, (w, h) in enumerate(_view_sizes(case, VIEW_SIZES[1:])):
            k = i % len(ids)
            info = resident[k].info()
            d = info.bounds_diagonal
            requests.append((ids[k], swr.make_camera(*_orbit(rng, info, w, h, 0.7 * d, 1.5 * d)), w, h))
        return {"case": case, "scenes": resident, "server": srv, "requests": requests, "held": [], "seen": {}}
    if kind == "noalloc":
        w, h = case["width"], case["height"]
        scene = swr.Scene(scenes.spheres_scene(seed=seed, count=case["objects"], subdiv=case["subdiv"], box=4.0,
                                               voxel=64))
        cam = swr.make_camera(*_orbit(rng, scene.info(), w, h, 8.0, 16.0))
        return {"case": case, "scene": scene, "cam": cam,
                "rgba": torch.zeros(h, w, dtype=torch.int32, device="cuda"),
                "vis": torch.zeros(h, w, dtype=torch.int64, device="cuda")}
    sd = scenes.textured_scene(seed=seed, count=case["objects"], subdiv=case["subdiv"], tex_size=16,
                               cube_size=case["cube"], voxel=case["voxel"])
    sd = _big_textures(sd, seed, case["tex"])
    sd["specular_samples"], sd["brdf_lut_size"] = 64, 128
    return {"case": case, "sd": sd, "scene": None}


# -------------------------------------------------------------------- calls


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "frame":
        r = state["r"]
        r.render(state["scene"], state["cam"], case["dt"])
        r.blit(state["pixels"])
        out = {"rgba8": state["frame"], "vis": state["vis"]}
        if case["dt"] > 0.0:
            out["exposure"] = r.exposure()
        return out
    if kind in ("batch_views", "batch_scenes"):
        state["batch"].render(state["views"])
        state["batch"].sync()
        return {"rgba8": state["rgba"], "vis": state["vis"]}
    if kind == "serve":
        return _serve(state)
    if kind == "noalloc":
        swr.check(swr.lib().swr_render_frame_noalloc(
            state["scene"].handle, C.byref(state["cam"]), case["width"], case["height"], 2.0, swr.RSQRT_AARCH64,
            C.c_void_p(state["rgba"].data_ptr()), C.c_void_p(state["vis"].data_ptr()), None))
        return {"rgba8": state["rgba"], "vis": state["vis"]}
    return _load(state)


def _serve(state):
    """Submits the burst and collects every frame; the last burst's framebuffers go back to the pool first."""
    srv, requests = state["server"], state["requests"]
    for ticket in state["held"]:
        srv.release(ticket)
    for i, (scene, cam, w, h) in enumerate(requests):
        srv.submit(scene, cam, w, h, tag=i)
    done = [None] * len(requests)
    state["held"], left = [], len(requests)
    while left:
        for c in srv.poll(len(requests), wait_ms=50):
            if c.status:
                raise RuntimeError("request %d: status %d" % (c.tag, c.status))
            done[c.tag] = c
            state["held"].append(c.ticket)
            left -= 1
    out = []
    for c in done:
        key = (c.rgba8, c.width, c.height)
        if key not in state["seen"]:
            state["seen"][key] = (_view_of(c.rgba8, (c.height, c.width), "<i4", srv)[:c.height & ~1],
                                  _view_of(c.vis, (c.height, c.width), "<i8", srv))
        out.append(state["seen"][key])
    return out


def _load(state):
    """Opens the scene and looks at the tables it holds; the scene stays open until the next pass."""
    if state["scene"] is not None:
        state["scene"].close()
    s = state["scene"] = swr.Scene(state["sd"], gi=state["case"]["gi"])
    e = s.export()

    def table(t):
        return _host_view(t.data, t.data_len, np.int32, s)

    def floats(ptr, n):
        return _host_view(ptr, n, np.float32, s) if ptr else None

    n = e.voxel_size ** 3
    prims = [e.primitives[i] for i in range(e.primitive_count)]
    return {"textures": [table(e.textures[i]) for i in range(e.texture_count)], "specular": table(e.cubemap_specular),
            "brdf_lut": table(e.brdf_lut), "irradiance": np.array(e.irradiance_sh),
            "sun": floats(e.voxel_light_intensity, n), "gi": floats(e.voxel_gi_sh4, n * 16),
            "normals": [floats(p.normals, p.vertex_count * 3) for p in prims],
            "tangents": [floats(p.tangents, p.vertex_count * 4) for p in prims]}


# --------------------------------------------------------------------- work

# Bytes a triangle's geometry takes (three indices, half a vertex of position,
# normal and texture coordinate) and a pixel's outputs (RGBA8 and visibility).
TRI_BYTES, PIXEL_BYTES = 12 + 16, 4 + 8
# Operations of the frame's formulas: three vertex transforms (79 each) and
# the triangle's setup; interpolation, normalisations, voxel light, BRDF,
# environment and tone map of a pixel (the baked grid interpolates 16 values).
TRI_FLOPS, PIXEL_FLOPS, GI_PIXEL_FLOPS = 350, 600, 800


def _sphere_tris(case):
    return case["objects"] * 20 * 4 ** case["subdiv"]


def work(case):
    kind = case["kind"]
    texels = case.get("textures", 1) * case.get("tex", 256) ** 2 * 4
    if kind in ("frame", "noalloc"):
        px = case["width"] * case["height"]
        tris = case["triangles"] if case.get("scene") == "stress" else _sphere_tris(case)
        slots = 5 if case.get("slots") else 1
        flops = tris * TRI_FLOPS + px * (GI_PIXEL_FLOPS if case.get("gi") else PIXEL_FLOPS)
        return {"bytes": tris * TRI_BYTES + px * PIXEL_BYTES + min(texels, px * 4) * slots, "flops": flops}
    if kind == "batch_views":
        px = sum(w * h for w, h in _view_sizes(case, VIEW_SIZES))
        tris = _sphere_tris(case)
        return {"bytes": tris * TRI_BYTES + px * PIXEL_BYTES + texels,
                "flops": tris * case["views"] * TRI_FLOPS + px * PIXEL_FLOPS}
    if kind == "batch_scenes":
        px, tris = sum(w * h for w, h in _view_sizes(case, SCENE_SIZES)), sum(_scene_sizes(case))
        return {"bytes": tris * TRI_BYTES + px * PIXEL_BYTES + min(texels * case["scenes"], px * 4),
                "flops": tris * TRI_FLOPS + px * PIXEL_FLOPS}
    if kind == "serve":
        px, tris = sum(w * h for w, h in _view_sizes(case, VIEW_SIZES[1:])), _scene_sizes(case)
        seen = sum(tris[i % len(tris)] for i in range(case["requests"]))
        return {"bytes": sum(tris) * TRI_BYTES + px * PIXEL_BYTES + min(texels * case["scenes"], px * 4),
                "flops": seen * TRI_FLOPS + px * PIXEL_FLOPS}
    # A load: textures in and mip chains out, geometry in and processed, the
    # prefiltered environment, the voxel grid; 64 samples of about 40
    # operations per environment texel, 64 rays of about 300 per baked voxel.
    tris, voxels = _sphere_tris(case), case["voxel"] ** 3
    env = 6 * case["cube"] ** 2 * (1 + int(math.log2(case["cube"])))
    size = 6 * case["tex"] ** 2 * 4 * 7 // 3 + tris * 64 + env * 4 + voxels * (64 if case["gi"] else 4)
    return {"bytes": size, "flops": env * 64 * 40 + (voxels * 64 * 300 // 8 if case["gi"] else voxels * 100)}


def exact(case, seed):
    """Frames are whole numbers (RGBA8, triangle IDs); the floating tables of a load come out of ray casts and
    texture filters that have no short form in 64 bits."""
    return None
