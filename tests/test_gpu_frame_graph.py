"""A renderer replays its launch sequence as a graph once a frame's arguments
have stayed the same for a few frames. Loops that cross that point, with the
camera moving, scenes alternating (opaque, translucent, baked light), exposure
steps in between and a blit target set and cleared, must give the frames of a
renderer that draws each of them first."""
import numpy as np
import pytest

import scenes
import swr

pytestmark = pytest.mark.gpu
W, H = 210, 130


@pytest.fixture(scope="module")
def three():
    s = [swr.Scene(scenes.small_scene(seed=4)), swr.Scene(scenes.translucent_scene(seed=4, count=4)),
         swr.Scene(scenes.small_scene(seed=6), gi=True)]
    yield s
    for x in s:
        x.close()


def camera(s, i):
    pos, at, fov, w, h, far = scenes.default_camera_params(s.info(), W, H)
    return swr.make_camera((pos[0] + 0.1 * i, pos[1], pos[2] - 0.05 * i), at, fov, w, h, far)


def fresh(s, cam):
    r = swr.Renderer(W, H)
    r.render(s, cam)
    out = r.blit(), r.visbuffer()
    r.close()
    return out


@pytest.mark.parametrize("order", [[0] * 12, [0] * 7 + [1] * 8 + [0] * 3, [2] * 6 + [0, 2, 1, 0] + [2] * 7])
def test_replayed_frames(three, order):
    r = swr.Renderer(W, H)
    launches, steps = 0, []
    for i, k in enumerate(order):
        cam = camera(three[k], i)
        r.render(three[k], cam)
        rgba, vis = r.blit(), r.visbuffer()
        want_rgba, want_vis = fresh(three[k], cam)
        assert np.array_equal(vis, want_vis) and np.array_equal(rgba, want_rgba), i
        steps.append((k, r.stats().kernel_launches - launches))
        launches = r.stats().kernel_launches
    for k in set(order):  # every frame of a scene counts the same kernels, replayed or not
        assert len({n for j, n in steps if j == k}) == 1, steps
    r.close()


def test_exposure_and_blit_target_between_replays(three):
    r, host = swr.Renderer(W, H), np.zeros((H, W), np.uint32)
    for i in range(16):
        cam = camera(three[0], i)
        if i in (6, 11):
            r.render(three[0], cam, 0.1)  # an exposure step: not the replayed sequence
            r.blit()
            r.set_exposure(2.0)
        r.set_blit_target(host.ctypes.data, W, keep=host) if i in (8, 9, 13) else r.set_blit_target(None)
        r.render(three[0], cam)
        rgba = r.blit(host) if i in (8, 9, 13) else r.blit()
        want_rgba, want_vis = fresh(three[0], cam)
        assert np.array_equal(rgba, want_rgba) and np.array_equal(r.visbuffer(), want_vis), i
    r.close()


@pytest.mark.parametrize("warm", [2, 8])
def test_frame_captured_by_the_caller(three, warm):
    """A stream that the caller captures gets the kernels themselves, before and after the renderer replays."""
    torch = pytest.importorskip("torch")
    r, s = swr.Renderer(W, H), torch.cuda.Stream()
    for i in range(warm):
        r.render(three[0], camera(three[0], i), stream=s.cuda_stream)
        r.blit(stream=s.cuda_stream)
    graph = torch.cuda.CUDAGraph()
    cam = camera(three[0], 3)
    with torch.cuda.graph(graph, stream=s, capture_error_mode="relaxed"):
        r.render(three[0], cam, stream=s.cuda_stream)
    for _ in range(2):
        graph.replay()
    torch.cuda.synchronize()
    want_rgba, want_vis = fresh(three[0], cam)
    assert np.array_equal(r.visbuffer(), want_vis) and np.array_equal(r.blit(), want_rgba)
    r.close()
